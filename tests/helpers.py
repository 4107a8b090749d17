"""Shared helpers for the tests: golden loading and seeded inputs."""
from __future__ import annotations

from pathlib import Path

import numpy as np
import torch

GOLDEN = Path(__file__).resolve().parent / "golden"


def load_golden(name: str):
    z = np.load(GOLDEN / f"{name}.npz")
    meta = z["meta"].tolist()
    world, B, S, H, hkv, D, seed = meta[:7]
    mesh = tuple(meta[7:])
    t = {k: torch.from_numpy(z[k]) for k in z.files if k != "meta"}
    return dict(world=world, B=B, S=S, H=H, hkv=hkv, D=D, seed=seed, mesh=mesh, t=t)


def golden_text(name: str) -> str:
    return (GOLDEN / f"{name}.gen.txt").read_text()


def shard_inputs(q, k, v, world):
    qs = [x.contiguous() for x in q.chunk(world, 1)]
    kvs = [torch.stack([k.chunk(world, 1)[r], v.chunk(world, 1)[r]]).contiguous() for r in range(world)]
    return qs, kvs


def seeded_qkv(seed, B, S, H, hkv, D, scale=0.5, dtype=torch.bfloat16, device="cpu"):
    """Q/K/V (and dO) ~ N(0,1)*scale from per-tensor seeds, built on the CPU then moved."""
    out = []
    for i, (heads) in enumerate((H, hkv, hkv, H)):
        g = torch.Generator().manual_seed(seed + i)
        out.append((torch.randn(B, S, heads, D, generator=g) * scale).to(dtype).to(device))
    return out


# Error bounds of the kernels, element by element.  What they round: the probabilities (and, backward, dS) to bf16 before
# a product that is summed in fp32, and the result to bf16.  Each rounding is off by at most 2^-8 of the value, so a result
# sum_j w_j x_j is off by at most 2^-8 (sum_j |w_j x_j| + |result|).  5 % more for the exponentials and the fp32
# sums (tensor cores truncate: 2^-23 of the sum of absolute values per 16 terms, 1 % of the bound at 4 096 keys).
def rounding_bound(mass: torch.Tensor, value: torch.Tensor) -> torch.Tensor:
    return 1.05 * 2.0 ** -8 * (mass + value.abs()) + 1e-6


def fwd_exact_and_mass(q, k, v, scale, causal=False, q_off=None):
    """Attention in fp32 and sum_j p_j |v_j|, both [B, Sq, Hq, D]."""
    from oracle import block

    o, _ = block.block_attn_fwd(q.float(), k, v, scale, causal=causal, q_off=q_off)
    mass, _ = block.block_attn_fwd(q.float(), k, v.abs(), scale, causal=causal, q_off=q_off)
    return o, mass


def bwd_mass(do, q, k, v, o, lse, scale, causal=False, q_off=0):
    """scale * sum_k |dS| |k|, scale * sum_q |dS| |q| and sum_q P |dO|: the masses of dq, dk and dv."""
    b, sq, hq, d = q.shape
    sk, hkv = k.shape[1], k.shape[2]
    heads = [x.float().permute(0, 2, 1, 3) for x in (do, q, o)]
    kf, vf = (x.float().permute(0, 2, 1, 3).repeat_interleave(hq // hkv, dim=1) for x in (k, v))
    dof, qf, of = heads
    s = qf @ kf.transpose(-1, -2) * scale
    if causal:
        hidden = torch.arange(sk)[None, :] > torch.arange(sq)[:, None] + q_off
        s = s.masked_fill(hidden, float("-inf"))
    p = torch.exp(s - lse.float().unsqueeze(-1)).nan_to_num(nan=0.0, posinf=0.0)
    ds = (p * (dof @ vf.transpose(-1, -2) - (dof * of).sum(-1, keepdim=True))).abs()
    mq = ds @ kf.abs() * scale
    mk, mv = ds.transpose(-1, -2) @ qf.abs() * scale, p.transpose(-1, -2) @ dof.abs()
    mk, mv = (x.reshape(b, hkv, hq // hkv, sk, d).sum(2) for x in (mk, mv))
    return tuple(x.permute(0, 2, 1, 3) for x in (mq, mk, mv))
