"""RoPE helpers and the host-side bit allocation of the K compressor.

Mirrors the parts of the reference's src/shard/rope.py that the compressed-KV
path uses.  The heavy lifting (RoPE removal over a whole prefill, the int4
quantiser) lives in CUDA; what is here is host control logic and the small
torch expressions of the non-fused read path.
"""
from __future__ import annotations

import ctypes as C
from operator import index

import torch

from . import _lib


def rotate_half(x):
    """HF Llama convention: (x1, x2) -> (-x2, x1) on the two halves of the last dim."""
    half = x.shape[-1] // 2
    return torch.cat([-x[..., half:], x[..., :half]], dim=-1)


def rope_cos_sin(positions, inv_freq):
    """cos/sin tables (T, hd) of fp32(pos) * fp32(inv_freq) duplicated over both halves."""
    ph = positions.to(torch.float32)[:, None] * inv_freq.to(positions.device, torch.float32)[None, :]
    emb = torch.cat([ph, ph], dim=-1)
    return emb.cos(), emb.sin()


def reapply_rope(keys, positions, inv_freq):
    """keys (..., T, hd) -> keys with RoPE at `positions` (reference: rope.py:26-30)."""
    cos, sin = rope_cos_sin(positions, inv_freq)
    return keys * cos + rotate_half(keys) * sin


def get_rope_inv_freq(model):
    """Find the model's rotary inv_freq table, else derive it from the config
    (reference: src/shard/rope.py:32-47)."""
    backbone = getattr(model, "model", getattr(model, "transformer", None))
    candidates = [backbone]
    layers = getattr(backbone, "layers", None) if backbone is not None else None
    if layers is not None and len(layers) > 0:
        candidates.append(layers[0])
    for owner in candidates:
        if owner is None:
            continue
        rot = getattr(owner, "rotary_emb", None)
        if rot is None:
            attn = getattr(owner, "self_attn", None)
            rot = getattr(attn, "rotary_emb", None) if attn is not None else None
        if rot is not None and hasattr(rot, "inv_freq"):
            return rot.inv_freq.detach().float().cpu()
    cfg = model.config
    hd = getattr(cfg, "head_dim", cfg.hidden_size // cfg.num_attention_heads)
    theta = getattr(cfg, "rope_theta", 10000.0)
    params = getattr(cfg, "rope_parameters", None)
    if isinstance(params, dict) and "rope_theta" in params:
        theta = params["rope_theta"]
    return 1.0 / (theta ** (torch.arange(0, hd, 2, dtype=torch.float32) / hd))


_GROUP = 64                 # components share a bit width in groups of 64


def dp_bit_allocation(variances, total_budget):
    """Bits per PCA component by dynamic programming (reference: rope.py:49-84).

    The programme itself runs in the library (host code).  Minimises sum_g err(g, bits_g) subject to
    sum_g ceil(size_g * bits_g / 16) <= total_budget // 16 + 1, with err = 4 * var for 0 bits and
    var / (3 * 4**bits) otherwise.  Ties keep the first (smallest) option.
    """
    v = variances.float().cpu()
    d = int(v.shape[0])
    n_groups = (d + _GROUP - 1) // _GROUP
    sizes = [min(_GROUP, d - g * _GROUP) for g in range(n_groups)]
    if n_groups == 0:
        return []
    gvar = [v[g * _GROUP: g * _GROUP + sizes[g]].sum().item() for g in range(n_groups)]
    bits = (C.c_int32 * n_groups)()
    _lib.check(_lib.load().shard_b200_dp_bit_allocation((C.c_double * n_groups)(*gvar), (C.c_int32 * n_groups)(*sizes), n_groups,
                                                        min(index(total_budget), 16 * d), bits), "dp_bit_allocation")
    alloc = []
    for g in range(n_groups):
        alloc += [bits[g]] * sizes[g]
    return alloc
