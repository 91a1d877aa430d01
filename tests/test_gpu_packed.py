"""Packed token rows: batches from about 18,944 token rows on give rows only to each environment's slots up to its last live one.  The same
environments in slices of a few hundred take the full layout: forwards must agree bit for bit, gradients up to the order of fp32
sums, whatever the masks are."""
import ctypes as C

import pytest
import torch

from helpers import make_cfg, cuda_policy
from oracle import body_policy_oracle as bo
from oracle import policy_oracle as po

pytestmark = pytest.mark.gpu


def _masks(kind, envs, slots, gen):
    if kind == "none":
        return torch.zeros(envs, slots)
    if kind == "all":
        return torch.ones(envs, slots)
    if kind == "holes":                       # any subset: the last live slot decides
        return (torch.rand(envs, slots, generator=gen) < 0.3).float()
    if kind == "last":                        # one live slot, anywhere
        return torch.eye(slots)[torch.randint(0, slots, (envs,), generator=gen)]
    assert kind == "runs"                     # long runs of empty and of full environments
    return (torch.arange(envs)[:, None] // 700 % 2 * torch.ones(1, slots)).float()


def _obs(kind, envs, seed):
    gen = torch.Generator().manual_seed(seed)
    obs = po.make_obs(envs, seed)
    obs[:, po.OFF_MASK:po.OFF_MASK + 24] = _masks(kind, envs, 24, gen)
    return obs


SHAPES = [("cfg1", {}), ("recipe", {}), ("recipe", dict(value_residual=True)), ("cfg1", dict(n_heads=2, value_residual=True)), ("cfg1", dict(n_heads=2)),
          ("cfg4", {}), ("cfg4", dict(value_residual=True)), ("cfg1", dict(emb_ln=True, final_ln=True)), ("tiny", dict(trunk_arch="simbav2")),
          ("cfg2", dict(value_residual=True))]


@pytest.mark.parametrize("kind", ["none", "all", "holes", "last", "runs"])
@pytest.mark.parametrize("name,opts", SHAPES)
def test_forward_gives_the_bits_of_the_full_layout(name, opts, kind):
    cfg = make_cfg(name, name == "recipe", opts=dict(opts, n_blocks=2))
    m = cuda_policy(cfg, po.build_state_dict(cfg, 6))
    envs = 2600 if kind == "runs" else 1037
    obs = _obs(kind, envs, 41).cuda()
    for o in (obs, obs.half()):
        logits, value = m.forward_stacked(o)
        for lo in range(0, envs, 500):
            l, v = m.forward_stacked(o[lo:lo + 500])
            assert torch.equal(l, logits[lo:lo + 500]) and torch.equal(v, value[lo:lo + 500]), lo
    m.check_device()


@pytest.mark.parametrize("envs", [653, 654, 1024, 1025, 2357, 4736, 8193])
def test_sizes_around_the_line_and_pairs_of_ctas(envs):
    cfg = make_cfg("cfg1", opts=dict(n_blocks=2))
    m = cuda_policy(cfg, po.build_state_dict(cfg, 6))
    obs = po.make_obs(envs, 42, padded=True).cuda()
    logits, value = m.forward_stacked(obs)
    for lo in range(0, envs, 600):
        l, v = m.forward_stacked(obs[lo:lo + 600])
        assert torch.equal(l, logits[lo:lo + 600]) and torch.equal(v, value[lo:lo + 600]), lo


@pytest.mark.parametrize("kind", ["none", "holes", "runs"])
def test_counts_of_two_launches(kind):
    cfg = make_cfg("cfg1", opts=dict(n_blocks=2))
    m = cuda_policy(cfg, po.build_state_dict(cfg, 6))
    obs = _obs(kind, 4700, 53).cuda()
    logits, value = m.forward_stacked(obs)
    for lo in range(0, 4700, 600):
        l, v = m.forward_stacked(obs[lo:lo + 600])
        assert torch.equal(l, logits[lo:lo + 600]) and torch.equal(v, value[lo:lo + 600]), lo


@pytest.mark.parametrize("name,envs", [("cfg1", 1403), ("cfg2", 2401), ("cfg4", 701), ("cfg1", 4700)])
def test_a_captured_graph_counts_anew(name, envs):
    """The counts live on the device: a graph that was captured with one batch of masks replays any other."""
    cfg = make_cfg(name, opts=dict(n_blocks=2))
    m = cuda_policy(cfg, po.build_state_dict(cfg, 6))
    m.flatten_fp16()
    obs = po.make_obs(envs, 54, padded=True).cuda()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        m.forward_stacked(obs)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        logits, value = m.forward_stacked(obs)
    for kind in ("all", "none", "holes", "last", "all", "runs"):
        obs.copy_(_obs(kind, envs, 55))
        graph.replay()
        l, v = m.forward_stacked(obs.clone())
        assert torch.equal(l, logits) and torch.equal(v, value), kind
        l, v = m.forward_stacked(obs[:600].clone())
        assert torch.equal(l, logits[:600]) and torch.equal(v, value[:600]), kind
    m.check_device()


@pytest.mark.parametrize("name,blocks,envs", [("tiny", 2, 1306), ("tiny", 2, 1307), ("tiny", 2, 2600), ("tiny", 3, 654), ("tiny", 3, 1114), ("tiny", 3, 1115),
                                              ("cfg1", 2, 1114), ("cfg1", 2, 1115), ("cfg1", 2, 1306), ("cfg1", 2, 1307)])
def test_narrow_policies_around_their_lines(name, blocks, envs):
    cfg = make_cfg(name, opts=dict(n_blocks=blocks))
    m = cuda_policy(cfg, po.build_state_dict(cfg, 6))
    obs = po.make_obs(envs, 42, padded=True).cuda()
    logits, value = m.forward_stacked(obs)
    for lo in range(0, envs, 600):
        l, v = m.forward_stacked(obs[lo:lo + 600])
        assert torch.equal(l, logits[lo:lo + 600]) and torch.equal(v, value[lo:lo + 600]), lo


@pytest.mark.parametrize("name,opts", [("cfg1", {}), ("recipe", dict(value_residual=True)), ("cfg4", {})])
def test_all_live_in_long_runs(name, opts):
    """The attention kernel of packed rows works by tiles of four environments where every slot is live, and by rows where a single one
    is not."""
    cfg = make_cfg(name, opts=dict(opts, n_blocks=2))
    m = cuda_policy(cfg, po.build_state_dict(cfg, 6))
    obs = po.make_obs(2401, 47).cuda()
    for dead in (0, 1):
        obs[1700:1700 + dead, po.OFF_MASK + 23] = 0.0
        logits, value = m.forward_stacked(obs)
        for lo in range(0, 2401, 600):
            l, v = m.forward_stacked(obs[lo:lo + 600])
            assert torch.equal(l, logits[lo:lo + 600]) and torch.equal(v, value[lo:lo + 600]), (dead, lo)


@pytest.mark.parametrize("envs", [575, 1001, 2401])
def test_all_live_objects(native, envs):
    cfg = bo.named_config("cfg2")
    cfg.n_blocks = 2
    from test_gpu_body_policy import cuda_body_policy
    m = cuda_body_policy(cfg, bo.build_state_dict(cfg, 7))
    obs = bo.make_obs(envs, cfg, 50).cuda()
    for dead in (0, 1):
        obs[400:400 + dead, -1] = 0.0
        logits, value = m.forward_stacked(obs)
        for lo in range(0, envs, 500):
            l, v = m.forward_stacked(obs[lo:lo + 500])
            assert torch.equal(l, logits[lo:lo + 500]) and torch.equal(v, value[lo:lo + 500]), (dead, lo)
    assert native.lib.bsrl_device_status() == 0


@pytest.mark.parametrize("name", ["cfg1", "recipe", "cfg4"])
def test_not_a_number_stays_in_its_environment(name):
    cfg = make_cfg(name, opts=dict(n_blocks=2))
    m = cuda_policy(cfg, po.build_state_dict(cfg, 6))
    obs = _obs("holes", 1200, 43).cuda()
    clean_l, clean_v = m.forward_stacked(obs)
    bad = torch.arange(3, 1200, 7, device="cuda")
    obs[bad, po.OFF_MASK + 2] = float("nan")      # into the key bias, and through the attention into every row of the environment
    obs[bad[::2], po.OFF_NOTES:po.OFF_MASK] = float("inf")
    logits, value = m.forward_stacked(obs)
    good = torch.ones(1200, dtype=torch.bool, device="cuda")
    good[bad] = False
    assert torch.equal(logits[good], clean_l[good]) and torch.equal(value[good], clean_v[good])
    assert torch.isnan(logits[bad]).any(-1).any(-1).all()


def _region(native, m, envs, name):
    """A named intermediate of the last forward, or None where the batch has none of that name."""
    off, rows, cols, ld, dt = C.c_int64(), C.c_int64(), C.c_int64(), C.c_int64(), C.c_int32()
    rc = native.lib.bsrl_workspace_region(C.byref(m._cfg), envs, name, C.byref(off), C.byref(rows), C.byref(cols), C.byref(ld), C.byref(dt))
    if rc:
        return None
    ws = m._workspaces[(envs, m.critic_q.weight.device)][0]
    kind = {native.F32: torch.float32, native.I32: torch.int32}[dt.value]
    assert cols.value == ld.value
    return ws[off.value:off.value + rows.value * cols.value * 4].view(kind).view(rows.value, cols.value).clone()


@pytest.mark.parametrize("kind", ["none", "holes"])
@pytest.mark.parametrize("name,envs", [("cfg1", 1403), ("recipe", 701), ("cfg4", 701), ("recipe", 4700)])
def test_stream_regions(native, name, envs, kind):
    """x_packed laid out by row_start is x_resolved of the same environments below the line; each batch has one of the two."""
    cfg = make_cfg(name, name == "recipe", opts=dict(n_blocks=3))
    m = cuda_policy(cfg, po.build_state_dict(cfg, 6))
    obs = _obs(kind, envs, 52).cuda()
    m.forward_stacked(obs)
    x, start = _region(native, m, envs, b"x_packed"), _region(native, m, envs, b"row_start")
    assert _region(native, m, envs, b"x_resolved") is None
    mask = obs[:, po.OFF_MASK:po.OFF_MASK + 24] > 0
    rows = 5 + torch.where(mask.any(1), 24 - mask.flip(1).float().argmax(1), 0)
    assert torch.equal(start.view(-1).long(), torch.cat([rows.new_zeros(1), rows.cumsum(0)]))
    for lo in range(0, envs, 500):
        part = obs[lo:lo + 500]
        m.forward_stacked(part)
        n = part.shape[0]
        assert _region(native, m, n, b"x_packed") is None and _region(native, m, n, b"row_start") is None
        full = _region(native, m, n, b"x_resolved").view(n, 29, -1)
        there = torch.arange(29, device="cuda")[None, :] < rows[lo:lo + n, None]
        assert torch.equal(full[there], x[int(start[lo]):int(start[lo + n])]), lo


@pytest.mark.parametrize("name,envs", [("cfg1", 1403), ("cfg4", 701), ("cfg1", 300)])
def test_stage_profile_counts_the_rows_that_there_are(native, name, envs):
    cfg = make_cfg(name, opts=dict(n_blocks=2))
    m = cuda_policy(cfg, po.build_state_dict(cfg, 6))
    obs = po.make_obs(envs, 51, padded=True).cuda()
    m.forward_stacked(obs)
    native.check(native.lib.bsrl_profile_enable(1))
    m.forward_stacked(obs)
    torch.cuda.synchronize()
    stages = native.profile_read()
    native.check(native.lib.bsrl_profile_enable(0))
    d, F = cfg.embed, cfg.embed * cfg.ffn_mult
    # (the full layout's kernels compute the dead slots' rows too)
    rows = envs * 29 if envs < 654 else 5 * envs + int(obs[:, po.OFF_MASK:po.OFF_MASK + 24].sum())
    close = lambda a, b: abs(a - b) <= 1e-9 * b
    if name == "cfg4":
        assert close(stages["ffn_up_gemm"]["flops"], 2 * (rows + 5 * envs) * d * F)
        assert close(stages["ffn_down_gemm"]["bytes"], (rows + 5 * envs) * F * 2 + 2 * d * F * 2 + rows * d * 8 + 5 * envs * d * 6)
    else:
        assert close(stages["block_tail"]["flops"], 2 * (rows + 5 * envs) * (d * d + 2 * d * F))
        assert close(stages["encoder_fused"]["flops"], 2 * rows * d * (64 + d))


def _same(a, b):
    """The same bits, and not a number in the same places."""
    return torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(a.nan_to_num(nan=0.0), b.nan_to_num(nan=0.0))


@pytest.mark.parametrize("bad,shows", [([float("inf")], True), ([float("-inf"), float("inf")], True), ([7e4], True), ([float("nan")], False),
                                       ([float("nan"), float("inf")], False), ([6e4], False)])
@pytest.mark.parametrize("name,opts", [("cfg1", {}), ("recipe", {}), ("recipe", dict(game="flux")), ("cfg4", {}), ("cfg1", dict(emb_ln=True, final_ln=True)),
                                       ("cfg1", dict(n_blocks=1))])
def test_dead_slots_that_fp16_cannot_hold(name, opts, bad, shows):
    """What a dead slot holds shows in its environment's outputs in the full layout as soon as its encoding is not a number; without a
    row it shows all the same."""
    cfg = make_cfg(name, name == "recipe", opts=dict(dict(n_blocks=2), **opts))
    m = cuda_policy(cfg, po.build_state_dict(cfg, 6))
    envs = 1403
    obs = po.make_obs(envs, 48, padded=True).cuda()
    obs[:, po.OFF_MASK + 22:po.OFF_MASK + 24] = 0.0
    for i, v in enumerate(bad):
        obs[2::3, po.OFF_NOTES + 18 * 23 + 5 * i] = v
        obs[3::7, po.OFF_NOTES + 18 * 22 + 1 + 4 * i] = v
    logits, value = m.forward_stacked(obs)
    for lo in range(0, envs, 401):
        l, v = m.forward_stacked(obs[lo:lo + 401])
        assert _same(l, logits[lo:lo + 401]) and _same(v, value[lo:lo + 401]), lo
    if name != "recipe":                         # (the geometry of such a slot may be not a number, which the encoder's ReLU drops)
        assert bool(torch.isnan(logits[2]).any()) == shows
    m.check_device()


@pytest.mark.parametrize("kind", ["none", "all", "holes"])
@pytest.mark.parametrize("name,opts", [("cfg1", {}), ("recipe", dict(value_residual=True)), ("cfg4", {}), ("cfg1", dict(emb_ln=True, final_ln=True)),
                                       ("tiny", dict(trunk_arch="simbav2"))])
def test_gradients_equal_the_sum_over_slices(name, opts, kind):
    _gradients_equal_the_sum_over_slices(name, opts, kind, 701, 351)


def _gradients_equal_the_sum_over_slices(name, opts, kind, envs, part):
    """Per row the same arithmetic, so the difference is the order of fp32 sums over some 20 thousand rows (about 2^-24 sqrt(rows) =
    1e-5 of the terms' root sum of squares; the bound allows the atomics' order on top)."""
    cfg = make_cfg(name, name == "recipe", opts=dict(opts, n_blocks=2))
    m = cuda_policy(cfg, po.build_state_dict(cfg, 5))
    obs, act, up = _obs(kind, envs, 44).cuda(), po.make_actions(envs, cfg, 22).cuda(), po.make_upstream(envs, cfg, 23)

    def loss(s):
        _, lp, ent, val = m.get_action_and_value(obs[s], act[s])
        return ((up["logprob"][s].cuda() * lp).sum() + (up["entropy"][s].cuda() * ent).sum() + (up["value"][s].cuda() * val).sum()
                + (up["value_logits"][s].cuda() * m._value_logits).sum())

    with torch.enable_grad():
        # whatever the buffers held before must not show: rows of other environments, and not a number
        m.get_action_and_value(torch.full_like(obs, float("nan")), act)[1].sum().backward()
        m.zero_grad()
        loss(slice(0, envs)).backward()
        whole = {k: p.grad.clone() for k, p in m.named_parameters() if p.grad is not None}
        m.zero_grad()
        for lo in range(0, envs, part):
            loss(slice(lo, lo + part)).backward()
    m.check_device()
    top = max(float(g.norm()) for g in whole.values())
    for k, g in whole.items():
        assert float((m.get_parameter(k).grad - g).norm()) <= 1e-4 * float(g.norm()) + 1e-6 * top, k


@pytest.mark.parametrize("name,opts,envs,kind", [("cfg1", {}, 2401, "all"), ("cfg1", {}, 2401, "holes"), ("cfg1", dict(value_residual=True), 4500, "runs"),
                                                 ("cfg1", {}, 5300, "holes"), ("tiny", dict(trunk_arch="simbav2"), 1310, "holes")])
def test_gradients_of_larger_batches(name, opts, envs, kind):
    """Two counting launches, both forms of the attention, launches that no longer overlap: gradients against the sum over slices.  Up to 150
    thousand rows: 2^-24 sqrt(rows) = 2.3e-5 of the terms' root sum of squares, within the bound of the smaller batches."""
    _gradients_equal_the_sum_over_slices(name, opts, kind, envs, 600)


@pytest.mark.parametrize("forward", [0, 1])
@pytest.mark.parametrize("name,opts", [("cfg1", {}), ("recipe", dict(value_residual=True)), ("cfg4", {}), ("cfg1", dict(emb_ln=True, final_ln=True))])
def test_either_engine_reads_what_either_saved(native, name, opts, forward):
    """Whichever engine fills a save buffer, both backwards read it: the same operands, so they differ by the order of fp32 sums only
    (the bound of the sums over slices).  The forwards themselves round fp16 values to other sides, and with them a share of the
    ReLUs next to zero: gradients a few per cent apart (measured: up to 2 % of their norm, or 4 % of a thousandth of the largest)."""
    envs = 701
    cfg = make_cfg(name, name == "recipe", opts=dict(opts, n_blocks=2))
    m = cuda_policy(cfg, po.build_state_dict(cfg, 5))
    obs, act, up = _obs("holes", envs, 44).cuda(), po.make_actions(envs, cfg, 22).cuda(), po.make_upstream(envs, cfg, 23)

    def grads(fwd, bwd):
        m.zero_grad()
        m._workspaces.clear()                 # their size is the engine's
        try:
            with torch.enable_grad():
                native.lib.bsrl_set_engine(fwd)
                _, lp, ent, val = m.get_action_and_value(obs, act)
                loss = (up["logprob"].cuda() * lp).sum() + (up["entropy"].cuda() * ent).sum() + (up["value"].cuda() * val).sum()
                native.lib.bsrl_set_engine(bwd)
                loss.backward()
            torch.cuda.synchronize()
        finally:
            native.lib.bsrl_set_engine(0)
            m._workspaces.clear()
        return {k: p.grad.clone() for k, p in m.named_parameters() if p.grad is not None}

    one, other, default = grads(forward, 0), grads(forward, 1), grads(0, 0)
    m.check_device()
    top = max(float(g.norm()) for g in default.values())
    assert one.keys() == other.keys() == default.keys()
    for k, g in one.items():
        assert float((other[k] - g).norm()) <= 1e-4 * float(g.norm()) + 1e-6 * top, k
        assert float((default[k] - g).norm()) <= 5e-2 * float(g.norm()) + 5e-4 * top, k


@pytest.mark.parametrize("bad", [float("nan"), float("-inf"), 7e4, 6e4])
@pytest.mark.parametrize("name,heads,envs", [("cfg1", 4, 1503), ("cfg2", 8, 1203), ("cfg4", 8, 803), ("cfg2", 8, 19000)])
def test_dead_objects_that_fp16_cannot_hold(native, name, heads, envs, bad):
    cfg = bo.named_config(name)
    cfg.n_blocks, cfg.n_heads = 2, heads
    from test_gpu_body_policy import cuda_body_policy
    m = cuda_body_policy(cfg, bo.build_state_dict(cfg, 7))
    obs = bo.make_obs(envs, cfg, 49, padded=True)
    obs[4::7, -cfg.n_obj:] = 0.0                 # environments without a live object
    obs[:, -1] = 0.0
    obs[2::3, cfg.body_dim + cfg.n_obj * cfg.obj_dim - 1] = bad
    obs = obs.cuda()
    logits, value = m.forward_stacked(obs)
    part = 18944 // (1 + cfg.n_obj)
    for lo in range(0, min(envs, 4 * part), part):
        l, v = m.forward_stacked(obs[lo:lo + part])
        n = l.shape[0]
        assert _same(l, logits[lo:lo + n]) and _same(v, value[lo:lo + n]), lo
    assert bool(torch.isnan(logits[2]).any()) == (bad != 6e4)
    assert native.lib.bsrl_device_status() == 0


@pytest.mark.parametrize("kind", ["none", "all", "holes", "last", "runs"])
@pytest.mark.parametrize("name,heads", [("cfg1", 4), ("cfg2", 8), ("cfg4", 8), ("cfg2", 4), ("cfg1", 2)])
def test_body_token_layout(native, name, heads, kind):
    cfg = bo.named_config(name)
    cfg.n_blocks, cfg.n_heads = 2, heads
    from test_gpu_body_policy import cuda_body_policy
    m = cuda_body_policy(cfg, bo.build_state_dict(cfg, 7))
    envs = 1503 if kind != "runs" else 2600
    obs = bo.make_obs(envs, cfg, 45)
    obs[:, -cfg.n_obj:] = _masks(kind, envs, cfg.n_obj, torch.Generator().manual_seed(46))
    obs = obs.cuda()
    logits, value = m.forward_stacked(obs)
    part = 18944 // (1 + cfg.n_obj)
    for lo in range(0, envs, part):
        l, v = m.forward_stacked(obs[lo:lo + part])
        assert torch.equal(l, logits[lo:lo + part]) and torch.equal(v, value[lo:lo + part]), lo
    obs[::5, 3] = float("nan")
    l2, v2 = m.forward_stacked(obs)
    good = torch.arange(envs, device="cuda") % 5 != 0
    assert torch.equal(l2[good], logits[good]) and torch.equal(v2[good], value[good])
    assert native.lib.bsrl_device_status() == 0


@pytest.mark.parametrize("kind", ["none", "holes", "runs"])
@pytest.mark.parametrize("name,heads,envs", [("cfg1", 4, 4500), ("cfg2", 8, 4200), ("cfg2", 4, 4200)])
def test_body_token_layout_of_two_counting_launches(native, name, heads, envs, kind):
    cfg = bo.named_config(name)
    cfg.n_blocks, cfg.n_heads = 2, heads
    from test_gpu_body_policy import cuda_body_policy
    m = cuda_body_policy(cfg, bo.build_state_dict(cfg, 7))
    obs = bo.make_obs(envs, cfg, 56)
    obs[:, -cfg.n_obj:] = _masks(kind, envs, cfg.n_obj, torch.Generator().manual_seed(57))
    obs = obs.cuda()
    logits, value = m.forward_stacked(obs)
    part = 18944 // (1 + cfg.n_obj)
    for lo in range(0, envs, part):
        l, v = m.forward_stacked(obs[lo:lo + part])
        assert torch.equal(l, logits[lo:lo + part]) and torch.equal(v, value[lo:lo + part]), lo
    assert native.lib.bsrl_device_status() == 0
