"""C-ABI library on a host without a GPU: it loads, exports what the header declares, and its
host-side logic (configuration checks, parameter table, lane tables, sizes) is right.
No compute entry point is called here."""
import ctypes as C

import pytest
import torch

from helpers import make_cfg, po


def _cfg(native, cfg):
    return native.make_config(cfg.embed, cfg.n_heads, cfg.n_blocks, cfg.ffn_mult, cfg.trunk_dim,
                              cfg.trunk_hidden, cfg.value_bins, cfg.note_geo, cfg.head_gears,
                              cfg.z_asinh, cfg.value_vmax, cfg.eps)


def test_every_declared_symbol_is_exported(native):
    names = native.declared_symbols()
    assert len(names) >= 15
    for n in names:
        assert hasattr(native.lib, n), n
    assert native.lib.bsrl_abi_version() == 3


def test_token_lanes_match_oracle(native):
    for tok, name in enumerate(po.LEAD_ORDER):
        lanes = po.token_lanes(name)
        got = [native.lib.bsrl_token_lane(tok, k) for k in range(len(lanes))]
        assert got == lanes
        assert native.lib.bsrl_token_lane(tok, len(lanes)) == -1
    assert native.lib.bsrl_token_lane(5, 0) == -1


@pytest.mark.parametrize("name,geo", [("tiny", False), ("cfg1", True), ("cfg2", False), ("cfg4", False),
                                      ("recipe", True)])
def test_param_table_is_the_reference_state_dict(native, name, geo):
    cfg = make_cfg(name, geo)
    sd = po.build_state_dict(cfg, 0)
    table = native.param_table(_cfg(native, cfg))
    assert sorted(n for n, _, _ in table) == sorted(sd)
    for n, rows, cols in table:
        assert sd[n].numel() == rows * cols, n
        assert sd[n].shape[0] == rows, n


@pytest.mark.parametrize("name", ["cfg1", "cfg2", "cfg4"])
def test_mac_per_env_matches_oracle(native, name):
    cfg = make_cfg(name)
    assert native.lib.bsrl_mac_per_env(C.byref(_cfg(native, cfg))) == po.mac_per_env(cfg)


def test_sizes_grow_with_batch(native):
    c = _cfg(native, make_cfg("cfg2"))
    w1 = native.lib.bsrl_workspace_bytes(C.byref(c), 1024)
    w2 = native.lib.bsrl_workspace_bytes(C.byref(c), 2048)
    assert 0 < w1 < w2 <= 2 * w1 + 65536
    assert native.lib.bsrl_workspace_bytes(C.byref(c), 0) >= 0
    assert native.lib.bsrl_weights_bytes(C.byref(c)) > 2 * 5_000_000  # > fp16 copy of 5.7 M params


@pytest.mark.parametrize("name,geo,opts", [("tiny", False, None), ("cfg1", False, None), ("cfg2", False, dict(value_residual=True)),
                                           ("recipe", True, None), ("cfg4", False, None), ("cfg2", False, dict(final_ln=True))])
def test_a_workspace_serves_every_smaller_batch(native, name, geo, opts):
    """Callers allocate once for their largest batch: the size never falls from one batch to the next larger one, in particular
    not where the few-environment path and its hidden buffer end."""
    from beatsaberrl_b200.policy import NotePolicy
    c = NotePolicy(**make_cfg(name, geo, opts=opts).ref_kwargs())._cfg
    sizes = [native.lib.bsrl_workspace_bytes(C.byref(c), n) for n in range(200)]
    assert sizes[0] >= 0 and all(a <= b for a, b in zip(sizes, sizes[1:]))


@pytest.mark.parametrize("name,blocks,lines", [("tiny", 2, [1306]), ("tiny", 3, [653, 1114, 1306]), ("cfg1", 1, [1306]), ("cfg1", 2, [653, 1114, 1306]),
                                               ("recipe", 6, [653]), ("cfg2", 1, [653]), ("cfg4", 6, [653])])
def test_every_batch_has_one_form_of_the_stream(native, name, blocks, lines):
    """29 rows per environment below each line and packed rows above it, or the other way round: one of the two, inside the workspace, the
    row table beside the rows; the warp-MMA engine packs nothing."""
    c = _cfg(native, make_cfg(name, name == "recipe", opts=dict(n_blocks=blocks)))

    def region(n, what):
        off, rows, cols, ld, dt = C.c_int64(), C.c_int64(), C.c_int64(), C.c_int64(), C.c_int32()
        rc = native.lib.bsrl_workspace_region(C.byref(c), n, what, C.byref(off), C.byref(rows), C.byref(cols), C.byref(ld), C.byref(dt))
        assert rc in (0, -5), rc
        if rc:
            return None
        end = off.value + rows.value * ld.value * 4
        assert end <= native.lib.bsrl_workspace_bytes(C.byref(c), n)
        return off.value, end

    packed = False
    for n in [1, 100] + [n for line in lines for n in (line, line + 1)] + [4096, 4097, 65536]:
        packed ^= n - 1 in lines
        full, x, start = (region(n, what) for what in (b"x_resolved", b"x_packed", b"row_start"))
        if packed:
            assert full is None and (start[1] <= x[0] or x[1] <= start[0]), n
        else:
            assert x is None and start is None and full is not None, n
        native.lib.bsrl_set_engine(1)
        assert region(n, b"x_resolved") is not None and region(n, b"x_packed") is None
        native.lib.bsrl_set_engine(0)


def test_config_errors_are_reported(native):
    good = make_cfg("cfg1")
    c = _cfg(native, good)
    assert native.lib.bsrl_config_validate(C.byref(c)) == 0
    c.embed = 100                      # not a multiple of 32
    assert native.lib.bsrl_config_validate(C.byref(c)) == -5
    assert "embed" in native.last_error()
    c = _cfg(native, good)
    c.n_heads = 3                      # 128 % 3 != 0
    assert native.lib.bsrl_config_validate(C.byref(c)) == -2
    c = _cfg(native, good)
    c.head_gears[4] = 9
    assert native.lib.bsrl_config_validate(C.byref(c)) == -2
    assert "head_gears" in native.last_error()
    c = _cfg(native, good)
    c.z_asinh = 0.0
    assert native.lib.bsrl_config_validate(C.byref(c)) == -2
    assert native.lib.bsrl_config_validate(None) == -1
    assert native.lib.bsrl_workspace_bytes(C.byref(c), 8) == -1


def test_null_and_size_checks_come_before_any_launch(native):
    """Bad arguments must be refused on the host (no device is present here at all)."""
    c = _cfg(native, make_cfg("tiny"))
    lib = native.lib
    assert lib.bsrl_forward(C.byref(c), None, None, 0, 4, None, None, None, None, 0, None) == -1
    assert lib.bsrl_pack_weights(C.byref(c), None, 0, None, 0, None) == -1
    assert lib.bsrl_linear(None, None, None, None, None, 0, 0, 8, 8, 32, 0, None) == -1
    fake = C.c_void_p(4096)            # never dereferenced: checks fail first
    assert lib.bsrl_linear(fake, fake, None, None, fake, 0, 0, 8, 8, 33, 0, None) == -2
    assert lib.bsrl_linear(C.c_void_p(4100), fake, None, None, fake, 0, 0, 8, 8, 32, 0, None) == -3
    assert lib.bsrl_attention(fake, fake, 4, 80, 2, 0, 29, fake, None) == -5   # head_dim 40
    assert lib.bsrl_attention(fake, fake, 4, 64, 2, 27, 5, fake, None) == -2   # queries past row 29
    # a workspace one byte short is refused
    need = lib.bsrl_workspace_bytes(C.byref(c), 4)
    assert lib.bsrl_forward(C.byref(c), C.c_void_p(256), fake, 0, 4, fake, fake, None,
                            C.c_void_p(512), need - 1, None) == -4


def test_policy_facade_host_side(native):
    from beatsaberrl_b200.policy import NotePolicy, bump_weights_version
    cfg = make_cfg("tiny", True, (5,) * 8 + (7,) + (5,) * 20)
    torch.manual_seed(9)
    m = NotePolicy(**cfg.ref_kwargs())
    sd = po.build_state_dict(cfg, 9)
    msd = m.state_dict()
    assert set(msd) == set(sd)
    for k in sd:                        # same creation order -> same seeded init as the reference
        assert torch.equal(msd[k], sd[k]), k
    assert m.k_max == 7 and m.n_lead == 5 and m.arch["head_gears"][8] == 7
    assert m.mac_per_env() == po.mac_per_env(cfg)
    with pytest.raises(RuntimeError):   # no CPU path
        m.forward_stacked(torch.zeros(2, 630))
    acc = NotePolicy(fp16_accum="all")      # a permission for cuBLAS in the reference: accepted, recorded, fp32 accumulation kept
    assert acc.arch["fp16_accum"] == "all" and acc.fp16_accum == "all"
    with pytest.raises(ValueError):
        NotePolicy(fp16_accum="sometimes")
    with pytest.raises(ValueError):
        NotePolicy(trunk_arch="mlp")
    with pytest.raises(ValueError):
        NotePolicy(z_asinh=0.0)
    bump_weights_version()


def test_a_replaced_module_is_the_one_that_gets_gradients(native):
    """The grad-mode forward hands the live parameters to autograd: after a module was replaced (at any depth) or a
    parameter exchanged, the new ones."""
    from beatsaberrl_b200.policy import NotePolicy
    kw = dict(embed=64, trunk_dim=128, n_blocks=2, n_heads=2, n_gears=5, trunk_arch="simbav2")
    m, other = NotePolicy(**kw), NotePolicy(**kw)

    def check():
        named = dict(m.named_parameters())
        got = m._table_params()
        assert len(got) == len(m._param_table) and all(p is named[n] for p, (n, _, _) in zip(got, m._param_table))

    check()
    for change in (lambda: setattr(m, "critic_q", other.critic_q), lambda: m.blocks.__setitem__(0, other.blocks[0]),
                   lambda: setattr(m, "blocks", other.blocks), lambda: m.blocks[1].ffn.__setitem__(2, torch.nn.Linear(256, 64)),
                   lambda: setattr(m.heads[3], "weight", torch.nn.Parameter(torch.zeros(5, 128))),
                   lambda: setattr(m, "trunk_alpha", other.trunk_alpha)):
        change()
        check()


def test_optimizers_can_be_copied(native):
    """copy.deepcopy of an optimizer (with its policy) is an optimizer of the copy: its own moments, no addresses of the original."""
    import copy
    from beatsaberrl_b200.optim import PackedAdamW, PackedMuon
    from beatsaberrl_b200.policy import NotePolicy
    m = NotePolicy(embed=64, trunk_dim=128, n_blocks=2, n_heads=2, n_gears=5)
    for opt, state in ((PackedAdamW(m), "exp_avg"), (PackedMuon(m), "bufs")):
        twin = copy.deepcopy(opt)
        live = dict(twin.policy.named_parameters())
        assert twin.policy is not m and all(p is live[n] for n, p in zip(twin.names, twin.params))
        getattr(twin, state)[0].fill_(1.0)
        assert float(getattr(opt, state)[0].abs().max()) == 0.0


def test_a_learning_rate_changed_in_place_is_seen(native):
    """Schedules may hold the rate in a tensor or an array and change that: the per-parameter rates follow its value."""
    import numpy as np
    from beatsaberrl_b200.optim import PackedAdamW, _lr_table
    from beatsaberrl_b200.policy import NotePolicy
    opt = PackedAdamW(NotePolicy(embed=64, trunk_dim=128, n_blocks=2, n_heads=2, n_gears=5))
    for rate, mult in ((torch.tensor(0.5), 2.0), (np.array(0.5), 2.0), (0.5, torch.tensor(2.0))):
        opt.lr, opt.lr_scale = rate, {"critic_": mult}
        assert set(_lr_table(opt, opt.names)[0]) == {0.5, 1.0}
        for value in (rate, mult):
            if not isinstance(value, float):
                value *= 0.25
        assert set(_lr_table(opt, opt.names)[0]) == ({0.5, 0.25} if isinstance(rate, float) else {0.125, 0.25})
