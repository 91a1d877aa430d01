"""AdamW over a ``NotePolicy``'s fp32 masters whose step also refreshes the packed fp16 arena.

The reference trainer runs a fused Adam step and then ``bump_weights_version()``, after which the next
forward recasts the flat fp16 replica (python/train_batch.py:2847-2854, python/fp16_linear.py:236-246).
Here one call -- ``bsrl_adam_step_pack``, a handful of launches for the whole model -- updates the
masters in place and writes every updated value straight to its place(s) in the arena, so there is no
separate refresh pass and a captured rollout graph sees the new weights on its next replay.

Arithmetic and hyper-parameters are ``torch.optim.AdamW``'s; like the reference's ``--weight-decay``
(python/train_batch.py:276-290) the decoupled decay applies to parameters with two or more
dimensions only.  Parameters without a gradient (frozen, or owned by another optimizer such as the
reference's Muon half) are left alone and only re-scattered.

``PackedMuon`` is that other half (python/train_batch.py:797-968): Nesterov momentum, five quintic Newton-Schulz
steps towards the nearest orthogonal matrix, an RMS-matched step scale, on the hidden 2-D matrices only.  It is
one call of the library too (``bsrl_muon_step``): the products of all matrices run together on the tensor cores with
fp32 accuracy, and the last kernel writes the masters and their places in the arena.
"""
from __future__ import annotations

import ctypes as C
from array import array

import torch

from . import _native as nat


def _lr_of(opt, name: str) -> float:
    for prefix, mult in opt.lr_scale.items():
        if name.startswith(prefix):
            return opt.lr * mult
    return opt.lr


def _lr_table(opt, names, wd=None):
    """Per-parameter learning rates (and weight decays) as C arrays, rebuilt only when a setting they come from changed."""
    key = (float(opt.lr), float(opt.weight_decay), tuple((k, float(v)) for k, v in opt.lr_scale.items()))
    if opt._lr_key != key:
        n = len(names)
        opt._lr_arrays = ((C.c_float * n)(*[_lr_of(opt, nm) for nm in names]), (C.c_float * n)(*(wd or [0.0] * n)))
        opt._lr_key = key
    return opt._lr_arrays


def _pointers(tensors):
    """Their addresses as a C array (18 us for 152 tensors; converting one by one took 46)."""
    return (C.c_void_p * len(tensors)).from_buffer(array("Q", map(torch.Tensor.data_ptr, tensors)))


class PackedAdamW:
    def __init__(self, policy, lr: float = 3e-4, betas=(0.9, 0.999), eps: float = 1e-8,
                 weight_decay: float = 0.0, lr_scale: dict | None = None, exclude=()):
        """``lr_scale`` maps parameter-name prefixes to learning-rate multipliers (the reference
        trains its critic at 3x the actor's rate); ``exclude`` names parameters another optimizer owns
        (``muon_param_names``): their gradients are ignored here."""
        self.policy = policy
        self.exclude = frozenset(exclude)
        self.lr, self.betas, self.eps, self.weight_decay = float(lr), tuple(betas), float(eps), float(weight_decay)
        self.lr_scale = dict(lr_scale or {})
        self.step_count = 0
        named = dict(policy.named_parameters())
        self.names = [n for n, _, _ in policy._param_table]
        self.params = [named[n] for n in self.names]
        for p in self.params:
            if p.dtype is not torch.float32 or not p.is_contiguous():
                raise ValueError("PackedAdamW needs contiguous float32 parameters")
        self.exp_avg = [torch.zeros_like(p, memory_format=torch.preserve_format) for p in self.params]
        self.exp_avg_sq = [torch.zeros_like(p, memory_format=torch.preserve_format) for p in self.params]
        self._lr_key = self._lr_arrays = None
        self._owned_key, self._owned = None, ()

    def zero_grad(self, set_to_none: bool = True) -> None:
        for p in self.params:
            if p.grad is not None:
                if set_to_none:
                    p.grad = None
                else:
                    p.grad.zero_()

    @torch.no_grad()
    def step(self, inv_scale: torch.Tensor | None = None, found_inf: torch.Tensor | None = None) -> None:
        pol = self.policy
        dev = self.params[0].device
        if dev.type != "cuda":
            raise RuntimeError("PackedAdamW runs on a CUDA device only")
        pol._pack()                           # the arena exists and its padding is zero
        self.step_count += 1
        n = len(self.params)
        if self._owned_key != self.exclude:
            self._owned_key = frozenset(self.exclude)
            self._owned = [i for i, nm in enumerate(self.names) if nm not in self._owned_key]
        grads, keep = (C.c_void_p * n)(), []
        for i in self._owned:
            p = self.params[i]
            g = p.grad
            if g is None or not p.requires_grad:
                continue
            if not g.is_contiguous():
                g = g.contiguous()
                keep.append(g)
            grads[i] = g.data_ptr()
        lr, wd = _lr_table(self, self.names, [self.weight_decay if p.dim() >= 2 else 0.0 for p in self.params]
                           if self.weight_decay else None)
        for name, s in (("inv_scale", inv_scale), ("found_inf", found_inf)):
            if s is not None and (s.numel() != 1 or s.dtype is not torch.float32 or s.device != dev):
                raise ValueError(f"{name} must be a one-element float32 tensor on {dev}")
        with torch.cuda.device(dev):
            nat.check(nat.lib.bsrl_adam_step_pack(
                C.byref(pol._cfg), _pointers(self.params), grads, _pointers(self.exp_avg), _pointers(self.exp_avg_sq), n,
                lr, wd, self.betas[0], self.betas[1], self.eps, self.step_count,
                inv_scale.data_ptr() if inv_scale is not None else None,
                found_inf.data_ptr() if found_inf is not None else None,
                pol._arena.data_ptr(), pol._arena.numel(), torch.cuda.current_stream().cuda_stream))
        # the arena already holds the new weights: no version bump, no repack

    def state_dict(self) -> dict:
        return {"step": self.step_count,
                "exp_avg": {n: t.clone() for n, t in zip(self.names, self.exp_avg)},
                "exp_avg_sq": {n: t.clone() for n, t in zip(self.names, self.exp_avg_sq)}}

    def load_state_dict(self, sd: dict) -> None:
        self.step_count = int(sd["step"])
        for n, m, v in zip(self.names, self.exp_avg, self.exp_avg_sq):
            m.copy_(sd["exp_avg"][n])
            v.copy_(sd["exp_avg_sq"][n])


# Newton-Schulz coefficients (those of bsrl_muon_step), one (a, b, c) per step, applied as a x + b x^3 + c x^5 to the
# singular values of the normalised update: the published five-step schedule the reference adopted
# (python/train_batch.py:797-816).
MUON_NS_COEFS = ((4.0848, -6.8946, 2.9270),
                 (3.9505, -6.3029, 2.6377),
                 (3.7418, -5.5913, 2.3037),
                 (2.8769, -3.1427, 1.2046),
                 (2.8366, -3.0525, 1.2012))


def muon_param_names(policy, enc_hidden: bool = False) -> list:
    """The parameters Muon owns (python/train_batch.py:947-967): hidden 2-D matrices only.  The 29 heads, the critic's
    final value-bin layer, every bias / LayerNorm vector and the token encoders stay with Adam; with ``enc_hidden``
    the encoders' second layers move to Muon and only their input layers (``*_mlp.0``) stay."""
    enc = ("note_mlp", "saber_mlp", "torso_mlp", "leg_mlp")
    last_critic = f"critic_mlp.{len(policy.critic_mlp) - 1}.weight"
    names = []
    for n, p in policy.named_parameters():
        if p.ndim != 2 or n.startswith("heads.") or n == last_critic:
            continue
        if n.startswith(enc) and (not enc_hidden or ".0." in n):
            continue
        names.append(n)
    return names


def orthogonalize(stack: torch.Tensor, eps: float = 1e-7) -> torch.Tensor:
    """Five Newton-Schulz steps on a stack (k, m, n) of wide (m <= n) fp32 matrices: each is scaled to unit Frobenius
    norm and pushed towards the nearest orthogonal matrix; the iteration runs on the small (m, m) Gram matrix.  The
    plain statement of what ``bsrl_muon_step`` computes."""
    x = stack / (torch.linalg.vector_norm(stack, dim=(1, 2), keepdim=True) + eps)
    for a, b, c in MUON_NS_COEFS:
        gram = torch.bmm(x, x.transpose(1, 2))
        poly = torch.baddbmm(gram, gram, gram, beta=b, alpha=c)          # b s + c s s
        x = torch.baddbmm(x, poly, x, beta=a)                            # a x + (b s + c s s) x
    return x


class PackedMuon:
    def __init__(self, policy, names=None, lr: float = 0.02, momentum: float = 0.95, weight_decay: float = 0.0,
                 lr_scale: dict | None = None):
        """``names``: the parameters this optimizer owns (default ``muon_param_names(policy)``); pair it with
        ``PackedAdamW(policy, ..., exclude=names)`` for the rest."""
        self.policy = policy
        self.lr, self.momentum, self.weight_decay = float(lr), float(momentum), float(weight_decay)
        self.lr_scale = dict(lr_scale or {})
        named = dict(policy.named_parameters())
        self.table = [n for n, _, _ in policy._param_table]              # every parameter, the library's order
        self.all_params = [named[n] for n in self.table]
        self.names = list(names) if names is not None else muon_param_names(policy)
        for n in self.names:
            if n not in named or named[n].ndim != 2:
                raise ValueError(f"PackedMuon owns 2-D parameters only: {n}")
        self.params = [named[n] for n in self.names]
        self.bufs = [torch.zeros_like(p) for p in self.params]
        self._slot = {n: i for i, n in enumerate(self.table)}
        for p in self.params:
            if p.dtype is not torch.float32 or not p.is_contiguous():
                raise ValueError("PackedMuon needs contiguous float32 parameters")
        self._ws_key, self._ws_bytes = None, 0
        self._lr_key = self._lr_arrays = None

    def zero_grad(self, set_to_none: bool = True) -> None:
        for p in self.params:
            if p.grad is not None:
                p.grad = None if set_to_none else p.grad.zero_()

    @torch.no_grad()
    def step(self, found_inf: torch.Tensor | None = None) -> None:
        pol = self.policy
        dev = self.params[0].device
        if dev.type != "cuda":
            raise RuntimeError("PackedMuon runs on a CUDA device only")
        pol._pack()
        if found_inf is not None and (found_inf.numel() != 1 or found_inf.dtype is not torch.float32 or found_inf.device != dev):
            raise ValueError(f"found_inf must be a one-element float32 tensor on {dev}")
        n = len(self.table)
        grads, bufs, owned = (C.c_void_p * n)(), (C.c_void_p * n)(), (C.c_int32 * n)()
        keep = []
        for name, p, b in zip(self.names, self.params, self.bufs):
            g = p.grad
            if g is None or not p.requires_grad:
                continue
            slot = self._slot[name]
            if not g.is_contiguous():
                g = g.contiguous()
                keep.append(g)
            grads[slot], bufs[slot], owned[slot] = g.data_ptr(), b.data_ptr(), 1
        lrs, _ = _lr_table(self, self.table)
        if self._ws_key != bytes(owned):
            self._ws_bytes = nat.lib.bsrl_muon_workspace_bytes(C.byref(pol._cfg), owned, n)
            if self._ws_bytes < 0:
                raise nat.BsrlError(int(self._ws_bytes), nat.last_error())
            self._ws_key = bytes(owned)
        ws = torch.empty(self._ws_bytes, dtype=torch.uint8, device=dev)
        with torch.cuda.device(dev):
            nat.check(nat.lib.bsrl_muon_step(
                C.byref(pol._cfg), _pointers(self.all_params), grads, bufs, n, lrs,
                self.weight_decay, self.momentum, found_inf.data_ptr() if found_inf is not None else None,
                pol._arena.data_ptr(), pol._arena.numel(), ws.data_ptr(), ws.numel(),
                torch.cuda.current_stream().cuda_stream))

    def state_dict(self) -> dict:
        return {"momentum": self.momentum, "bufs": {n: b.clone() for n, b in zip(self.names, self.bufs)}}

    def load_state_dict(self, sd: dict) -> None:
        if set(sd["bufs"]) != set(self.names):
            raise ValueError("muon state does not match this policy's muon parameters")
        for n, b in zip(self.names, self.bufs):
            b.copy_(sd["bufs"][n])
