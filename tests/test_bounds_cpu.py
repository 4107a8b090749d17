"""The error bounds that the GPU tests use, on the CPU: results with the kernels' roundings keep them, results that lost a
part do not."""
import pytest
import torch

from oracle import block
from tests.helpers import bwd_mass, fwd_exact_and_mass, rounding_bound, seeded_qkv


def _bf16(x):
    return x.bfloat16().float()


@pytest.mark.parametrize("Sq,Sk,shares", [(1, 3001, 24), (100, 4096, 9), (60, 1400, 11)])
def test_forward_bound_notices_a_lost_share(Sq, Sk, shares):
    q, k, v, _ = seeded_qkv(11, 1, max(Sq, Sk), 2, 2, 128)
    q, k, v = q[:, :Sq], k[:, :Sk], v[:, :Sk]
    scale = 128 ** -0.5
    o, mass = fwd_exact_and_mass(q, k, v, scale)
    heads = [x.float().transpose(1, 2) for x in (q, k, v)]
    s = heads[0] @ heads[1].transpose(-1, -2) * scale
    p = torch.exp(s - s.max(-1, keepdim=True).values)
    lost = p.clone()
    lost[..., :Sk // shares] = 0                                  # one share's rows are missing, its sum is not
    bound = rounding_bound(mass, o)
    for weights, exceed in ((p, 0.0), (lost, 0.25)):
        got = _bf16((_bf16(weights) @ heads[2] / p.sum(-1, keepdim=True)).transpose(1, 2))
        over = ((got - o).abs() > bound).float()
        assert over.max() == 0 if exceed == 0 else over.mean() >= exceed
    # every single (row, head) would show it
    assert (over.amax(-1) == 1).all()


def test_backward_bound_notices_a_lost_key_tile():
    q, k, v, do = seeded_qkv(31, 1, 200, 2, 2, 128)
    q, do = q[:, :65], do[:, :65]
    scale = 128 ** -0.5
    ro, rl = block.block_attn_fwd(q, k, v, scale)
    dq, dk, dv = block.block_attn_bwd(do, q, k, v, ro, rl, scale)
    mq, mk, mv = bwd_mass(do, q, k, v, ro, rl, scale)
    one, _, _ = block.block_attn_bwd(do, q, k[:, :128], v[:, :128], ro, rl, scale)   # without the second tile
    over = (one - dq).abs() > rounding_bound(mq, dq)
    assert over.float().mean() >= 0.5 and (over.float().mean(-1) >= 0.25).all()
    # the roundings of the kernel keep it
    h = [x.float().transpose(1, 2) for x in (do, q, k, v, ro)]
    p = torch.exp(h[1] @ h[2].transpose(-1, -2) * scale - rl.unsqueeze(-1))
    ds = _bf16(p * (h[0] @ h[3].transpose(-1, -2) - (h[0] * h[4]).sum(-1, keepdim=True)))
    for got, want, mass in ((ds @ h[2] * scale, dq, mq), (ds.transpose(-1, -2) @ h[1] * scale, dk, mk),
                            (_bf16(p).transpose(-1, -2) @ h[0], dv, mv)):
        assert ((_bf16(got).transpose(1, 2) - want).abs() <= rounding_bound(mass, want)).all()
