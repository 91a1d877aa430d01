"""The work that users of this package have it do, as cases that can be timed and compared.

A case names one call pattern (``call``), one policy shape (``arch``, with ``blocks`` transformer blocks), a batch
(``envs``) and the options in use:

* ``forward``   logits and value of a batch of observations (viewer, replay evaluation, benchmarks);
* ``graphed``   the same behind ``GraphedForward``, as an evaluation loop at a fixed number of environments runs it;
* ``rollout``   one tick of the PPO rollout: sampled actions, with the trainer's buffer rows written on the way;
* ``evaluate``  log-probability, entropy and value of stored actions, without gradients;
* ``update``    one PPO minibatch: differentiable recompute, loss, backward, AdamW step with the weight refresh;
* ``optim``     one step of the hybrid optimizer (Muon on the hidden matrices, AdamW on the rest);
* ``body``      log-probability, entropy and value in the single-body-token layout.

Rollout buffers hold observations in fp16 and actions in uint8, so those are the inputs of ``evaluate`` and
``update``; the simulator hands over fp32 observations, the input of everything else.
"""
import math

import torch

from beatsaberrl_b200.body_policy import BodyObjectPolicy
from beatsaberrl_b200.graphs import GRAPH_WARMUP, GraphedForward
from beatsaberrl_b200.optim import PackedAdamW, PackedMuon, muon_param_names
from beatsaberrl_b200.policy import (NOTE_FEAT, N_ACTION_HEADS, N_NOTE_SLOTS, OBS_DIM, OFF_NOTE_MASK, OFF_NOTES,
                                     NotePolicy)

BINS = 101
T, LEAD = 29, 5

# The policy shapes of the benchmark and the tests: a small test policy, a two-block policy, the production shape, the
# benchmark's headline policy, and the wide one.
ARCHS = {
    "tiny": dict(embed=64, trunk_dim=128, n_blocks=2, n_heads=2, n_gears=5),
    "small": dict(embed=128, trunk_dim=256, n_blocks=2, n_heads=4, n_gears=5),
    "recipe": dict(embed=192, trunk_dim=384, n_blocks=6, n_heads=4, n_gears=5, note_geo=True),
    "headline": dict(embed=256, trunk_dim=512, n_blocks=4, n_heads=8, n_gears=5),
    "wide": dict(embed=512, trunk_dim=1024, n_blocks=6, n_heads=8, n_gears=7),
}
# The same in the single-body-token layout, with the object counts that go with them.
BODY_ARCHS = {
    "small": dict(embed=128, n_heads=4, n_blocks=2, n_obj=16, n_gears=5),
    "headline": dict(embed=256, n_heads=8, n_blocks=4, n_obj=32, n_gears=5),
    "wide": dict(embed=512, n_heads=8, n_blocks=6, n_obj=64, n_gears=7),
}
# Constructor options beyond the shape, as a training run switches them on.
OPTIONS = {
    "none": {},
    "norms": dict(emb_ln=True, final_ln=True),
    "vres": dict(value_residual=True),
    "simbav2": dict(trunk_arch="simbav2"),
}
MOST_ENVS = {"forward": 65536, "graphed": 4096, "rollout": 65536, "evaluate": 65536, "update": 16384, "body": 65536}
LEAST_ENVS = {"forward": 1, "graphed": 1, "rollout": 64, "evaluate": 64, "update": 64, "body": 1}
CALLS = ("forward", "graphed", "rollout", "evaluate", "update", "optim", "body")


def listed():
    return [
        # one environment: the viewer and replay tools step a trained policy tick by tick
        case("play_one_env", "forward", "recipe", 1),
        # evaluation over a few hundred maps at once, graph-replayed
        case("graphed_eval", "graphed", "recipe", 256),
        # a small training run's tick
        case("rollout_small", "rollout", "small", 1024),
        # the production run's tick
        case("rollout_recipe", "rollout", "recipe", 32768),
        # the benchmark's headline batch
        case("forward_headline", "forward", "headline", 65536),
        # the wide policy's batch
        case("forward_wide", "forward", "wide", 32768),
        # an odd tail of stored steps re-evaluated without gradients (KL and explained-variance diagnostics)
        case("evaluate_ragged", "evaluate", "headline", 5003),
        # the PPO update at the benchmark's minibatch
        case("update_headline", "update", "headline", 16384),
        # a small odd minibatch of the production shape with the value residual in use
        case("update_ragged", "update", "recipe", 2049, "vres"),
        # the optimizer half of an update alone, hybrid form
        case("optim_headline", "optim", "headline", 0),
        # single-body-token layout: its benchmark batch, and the wide form with 65 tokens at an odd batch
        case("body_headline", "body", "headline", 65536),
        case("body_wide", "body", "wide", 4095),
    ]


def case(name, call, arch, envs, options="none", blocks=0):
    blocks = blocks or (BODY_ARCHS if call == "body" else ARCHS)[arch]["n_blocks"]
    c = dict(call=call, arch=arch, blocks=blocks, envs=envs, options=options)
    return dict(c, name=name) if name else c


def shape(c):
    return dict((BODY_ARCHS if c["call"] == "body" else ARCHS)[c["arch"]], n_blocks=c["blocks"])


def draw(rng):
    call = rng.choice(CALLS)
    arch = rng.choice(sorted(BODY_ARCHS if call == "body" else ARCHS))
    blocks = rng.randint(2, 6)
    if call == "optim":
        return case("", call, arch, 0, rng.choice(sorted(OPTIONS)), blocks)
    options = rng.choice(sorted(OPTIONS)) if call != "body" and rng.random() < 0.3 else "none"
    lo, hi = LEAST_ENVS[call], MOST_ENVS[call]
    envs = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    top = max(flops_of(c) for c in listed())
    while envs > lo and flops_of(case("", call, arch, envs, options, blocks)) > top:
        envs = max(lo, envs // 2)
    return case("", call, arch, envs, options, blocks)


# ---------------------------------------------------------------- inputs
def make_obs(envs, gen):
    """Observations as the trainer's environments write them: N(0, 1) clipped to +-5, the first n of 24 note slots live
    (n uniform), dead slots zero, is_wall lanes 0 or 1."""
    obs = torch.randn(envs, OBS_DIM, generator=gen, device="cuda").clamp_(-5.0, 5.0)
    n = torch.randint(0, N_NOTE_SLOTS + 1, (envs, 1), generator=gen, device="cuda")
    mask = (torch.arange(N_NOTE_SLOTS, device="cuda")[None, :] < n).float()
    notes = obs[:, OFF_NOTES:OFF_NOTE_MASK].view(envs, N_NOTE_SLOTS, NOTE_FEAT)
    notes[:, :, 14] = (notes[:, :, 14] > 0.5).float()
    notes *= mask[:, :, None]
    obs[:, OFF_NOTE_MASK:OFF_NOTE_MASK + N_NOTE_SLOTS] = mask
    return obs


def make_body_obs(envs, arch, gen):
    """Single-body-token observations: 340 body lanes, n_obj objects of 16 lanes, n_obj live flags (first n live)."""
    n_obj = arch["n_obj"]
    obs = torch.randn(envs, 340 + 17 * n_obj, generator=gen, device="cuda").clamp_(-5.0, 5.0)
    n = torch.randint(0, n_obj + 1, (envs, 1), generator=gen, device="cuda")
    live = (torch.arange(n_obj, device="cuda")[None, :] < n).float()
    obs[:, 340:340 + 16 * n_obj].view(envs, n_obj, 16).mul_(live[:, :, None])
    obs[:, -n_obj:] = live
    return obs


def make_policy(c, seed):
    torch.manual_seed(seed)
    with torch.device("cuda"):
        if c["call"] == "body":
            policy = BodyObjectPolicy(**shape(c))
        else:
            policy = NotePolicy(**shape(c), **OPTIONS[c["options"]])
    policy.flatten_fp16()
    return policy


def prepare(case, seed):
    c = case
    policy = make_policy(c, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = dict(call=c["call"], policy=policy)
    B = c["envs"]
    if c["call"] == "optim":
        for p in policy.parameters():
            if p.requires_grad:
                p.grad = torch.randn(p.shape, generator=gen, device="cuda") * 0.01
        names = muon_param_names(policy)
        s["muon"] = PackedMuon(policy, names, lr=0.02, momentum=0.95)
        s["adam"] = PackedAdamW(policy, lr=3e-4, exclude=names, lr_scale={"critic_": 3.0})
        return s
    if c["call"] == "body":
        s["obs"] = make_body_obs(B, shape(c), gen)
    else:
        s["obs"] = make_obs(B, gen)
    gears = shape(c)["n_gears"]
    if c["call"] == "graphed":
        s["graph"] = GraphedForward(policy, B)
        for _ in range(GRAPH_WARMUP + 1):
            s["graph"](s["obs"])
    if c["call"] == "rollout":
        policy.seed_sampler(seed)
        s["rows"] = dict(b_act=torch.empty(B, N_ACTION_HEADS, dtype=torch.uint8, device="cuda"),
                         b_logp=torch.empty(B, device="cuda"), b_val=torch.empty(B, device="cuda"),
                         b_obs=torch.empty(B, OBS_DIM, dtype=torch.float16, device="cuda"),
                         ret_sig=torch.tensor(1.7, device="cuda"), ret_mu=torch.tensor(0.3, device="cuda"))
    if c["call"] in ("evaluate", "update", "body"):
        s["act"] = torch.randint(0, gears, (B, N_ACTION_HEADS), generator=gen, device="cuda").to(torch.uint8)
    if c["call"] in ("evaluate", "update"):
        s["obs"] = s["obs"].half()
    if c["call"] == "update":
        s["opt"] = PackedAdamW(policy, lr=3e-4, lr_scale={"critic_": 3.0})
        with torch.no_grad():
            s["old_logp"] = policy.get_action_and_value(s["obs"], s["act"])[1]
        s["adv"] = torch.randn(B, generator=gen, device="cuda")
        ret = torch.randn(B, 1, generator=gen, device="cuda")
        # HL-Gauss: the return as a Gaussian over the value bins
        s["target"] = torch.softmax(-0.5 * ((policy.value_centers - ret) / policy.value_sigma) ** 2, 1)
    return s


# ---------------------------------------------------------------- one pass
def run(state):
    s = state
    call, policy = s["call"], s["policy"]
    if call == "forward":
        with torch.no_grad():
            return policy.forward_stacked(s["obs"])
    if call == "graphed":
        return s["graph"](s["obs"])
    if call == "rollout":
        rows = s["rows"]
        action, logp, _, value = policy.rollout_step(s["obs"], **rows)
        return action, logp, value, rows["b_act"], rows["b_val"], rows["b_obs"]
    if call in ("evaluate", "body"):
        with torch.no_grad():
            _, logp, entropy, value = policy.get_action_and_value(s["obs"], s["act"])
        return logp, entropy, value, policy._ent_h
    if call == "update":
        _, logp, entropy, value = policy.get_action_and_value(s["obs"], s["act"])
        ratio = (logp - s["old_logp"]).exp()
        adv = s["adv"]
        pg = -torch.min(ratio * adv, ratio.clamp(0.8, 1.2) * adv).mean()
        vf = -(torch.log_softmax(policy._value_logits, 1) * s["target"]).sum(1).mean()
        loss = pg + 0.5 * vf - 0.001 * entropy.mean()
        s["opt"].zero_grad()
        loss.backward()
        s["opt"].step()
        params = s["opt"].params
        return (loss.detach(), logp.detach(), entropy.detach(), value.detach(),
                torch.cat([p.grad.reshape(-1) for p in params if p.grad is not None]),
                torch.cat([p.detach().reshape(-1) for p in params]))
    s["muon"].step()
    s["adam"].step()
    return [torch.cat([t.detach().reshape(-1) for t in ts])
            for ts in (s["adam"].params, s["muon"].bufs, s["adam"].exp_avg, s["adam"].exp_avg_sq)]


# ---------------------------------------------------------------- what a pass cannot do without
def params_of(c):
    """The parameters of the case's policy as (rows, columns); biases and norms in one piece."""
    if c["call"] == "body":
        a = shape(c)
        d, L = a["embed"], a["n_blocks"]
        mats = [(d, 340), (d, 16), (N_ACTION_HEADS * a["n_gears"], d), (1, d)]
    else:
        a = shape(c)
        d, L, D = a["embed"], a["n_blocks"], a["trunk_dim"]
        note = NOTE_FEAT + (22 if a.get("note_geo") else 0)
        mats = [(d, k) for k in (note, 49, 29, 34)] + [(d, d)] * 4
        mats += [(D, LEAD * d), (D, D), (D, D), (N_ACTION_HEADS * a["n_gears"], D)]
        mats += [(d, d)] * 4 + [(D, d + D), (D, D), (BINS, D)]
    return mats + [(d, d)] * (4 * L) + [(4 * d, d), (d, 4 * d)] * L


def macs_per_env(c):
    """Multiply-accumulates of one environment's forward: the last block serves its readout rows only."""
    if c["call"] == "body":
        a = shape(c)
        d, L, n = a["embed"], a["n_blocks"], a["n_obj"] + 1
        block, last = 12 * n * d * d + 2 * n * n * d, (2 * n + 10) * d * d + 2 * n * d
        return d * (340 + 16 * (n - 1)) + (L - 1) * block + last + d * (N_ACTION_HEADS * a["n_gears"] + 1)
    a = shape(c)
    d, L, D = a["embed"], a["n_blocks"], a["trunk_dim"]
    note = NOTE_FEAT + (22 if a.get("note_geo") else 0)
    encoders = d * (N_NOTE_SLOTS * note + 2 * 49 + 29 + 2 * 34) + T * d * d
    block, last = 12 * T * d * d + 2 * T * T * d, (2 * T + 10 * LEAD) * d * d + 2 * LEAD * T * d
    trunk = LEAD * d * D + 2 * D * D + D * N_ACTION_HEADS * a["n_gears"]
    critic = 2 * T * d * d + 2 * d * d + 2 * T * d + (d + D) * D + D * D + BINS * D
    return encoders + (L - 1) * block + last + trunk + critic


def flops_of(c):
    if c["call"] == "optim":     # five Newton-Schulz steps on the small side m of each hidden matrix: m m n, m m m, m m n
        a = shape(c)
        d, D, L = a["embed"], a["trunk_dim"], a["n_blocks"]
        hidden = [(d, d)] * (4 * L + 4) + [(d, 4 * d)] * (2 * L)
        hidden += [(D, LEAD * d), (D, D), (D, D), (D, d + D), (D, D)]
        return sum(10 * (2 * min(s) ** 2 * max(s) + min(s) ** 3) for s in hidden)
    return (6 if c["call"] == "update" else 2) * macs_per_env(c) * c["envs"]


def work(case):
    c = case
    n = sum(r * k for r, k in params_of(c))
    B = c["envs"]
    if c["call"] == "optim":     # master, gradient and momentum in; master, momentum and the fp16 copy out
        return {"bytes": n * 22, "flops": flops_of(c)}
    obs = (OBS_DIM if c["call"] != "body" else 340 + 17 * shape(c)["n_obj"]) * 4
    gears = shape(c)["n_gears"]
    per_env = {"forward": obs + 4 * (N_ACTION_HEADS * gears + 1), "graphed": obs + 4 * (N_ACTION_HEADS * gears + 1),
               "rollout": obs + OBS_DIM * 2 + N_ACTION_HEADS * 9 + 12,
               "evaluate": obs // 2 + N_ACTION_HEADS * 5 + 12, "body": obs + N_ACTION_HEADS * 5 + 12,
               "update": obs // 2 + N_ACTION_HEADS * 5 + 12 + 4 * (2 * BINS + 2)}[c["call"]]
    weights = n * (2 + 4 * 7 if c["call"] == "update" else 2)
    return {"bytes": B * per_env + weights, "flops": flops_of(c)}


def tolerance(case):
    """fp16 operands (11-bit significands) with fp32 sums throughout: two correct implementations that round in other
    places differ by a few 1e-3 in the outputs, by up to a share of 1e-3 in sampled near-ties, and by about one per cent
    more in gradients for the ReLUs near zero that fall to the other side.  The optimizer alone is fp32 arithmetic; its
    Newton-Schulz steps multiply a rounding by up to the product of their slopes at zero, (about 3.5) ** 5 = 500."""
    if case["call"] == "optim":
        return {"rel": 1e-5, "max": 1e-3}
    if case["call"] == "update":
        return {"rel": 2e-2}
    if case["call"] == "rollout":
        return {"rel": 1e-2, "differ": 5e-3}
    return {"rel": 5e-3}
