"""What is timed: attention work that programs on this library have it do, on one GPU.

Every case goes through a public entry point: `RingAttention` (the fused call, with and without its backward), the
per-step drop-ins that generated programs call (`_flash_attn_forward`, `_flash_attn_backward`, `update_out_and_lse`),
and `attn_fwd_segments` (one rank's ring in one launch, the shards in place).  bf16 with head_dim 128 is what the
library takes.  Inputs are N(0, 1) * 0.5, as in the benchmark and the tests.
"""
from __future__ import annotations

import math

import torch

import mercury_artifact_b200 as mb
from mercury_artifact_b200.ring import RingAttention

D = 128
SCALE = D ** -0.5

# (query heads, K/V heads): the layouts of the benchmark and of the tests
HEADS = ((32, 32), (16, 16), (8, 8), (32, 8), (16, 4), (8, 2), (4, 2))


def listed():
    return [
        # one block of a small test or of a toy model: launches and host work
        dict(name="block_small", kind="block", batch=1, sq=256, sk=256, hq=8, hkv=8, causal=False),
        # new tokens against a long context (bottom-right aligned causal block, Sq < Sk)
        dict(name="block_continue", kind="block", batch=1, sq=100, sk=16384, hq=32, hkv=8, causal=True),
        # the shape of the double-ring benchmark script, whole on one GPU
        dict(name="forward_8k", kind="forward", batch=1, seq=8192, hq=32, hkv=32, causal=False),
        # the headline workload
        dict(name="forward_32k", kind="forward", batch=1, seq=32768, hq=32, hkv=32, causal=True),
        # the target length with the grouped head layout: the largest call
        dict(name="forward_131k_gqa", kind="forward", batch=1, seq=131072, hq=32, hkv=8, causal=True),
        # a batch of odd length, grouped heads: inference prefill
        dict(name="forward_ragged", kind="forward", batch=2, seq=2999, hq=16, hkv=4, causal=True),
        # what one rank of eight computes of a 32768-token non-causal ring, shards in arrival order, one launch
        dict(name="ring_segments", kind="segments", batch=1, shards=8, shard=4096, hq=32, hkv=32, causal=False),
        # the generated program's loop over four shards: block call and running merge per step
        dict(name="ring_steps", kind="steps", batch=1, shards=4, shard=2048, hq=32, hkv=32, causal=False),
        # the block call of the generated backward loop
        dict(name="block_backward", kind="block_backward", batch=1, sq=4096, sk=4096, hq=32, hkv=32, causal=False),
        # forward and backward of a small model
        dict(name="train_1k", kind="train", batch=2, seq=1024, hq=8, hkv=8, causal=True, deterministic=False),
        # forward and backward of the headline workload
        dict(name="train_32k", kind="train", batch=1, seq=32768, hq=32, hkv=32, causal=True, deterministic=False),
        # bitwise reproducible training, odd length, grouped heads
        dict(name="train_deterministic", kind="train", batch=1, seq=6001, hq=32, hkv=8, causal=True, deterministic=True),
    ]


def _log_size(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    # a third as they come (odd ones among them), the others in the multiples that programs use
    step = rng.choice((1, 64, 128)) if n >= 256 else 1
    return max(lo, n // step * step)


def draw(rng):
    largest = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(("block", "continue", "forward", "segments", "steps", "block_backward", "train", "train"))
        hq, hkv = rng.choice(HEADS)
        batch = rng.choice((1, 1, 2, 4))
        causal = rng.random() < 0.6
        c = dict(kind=kind, batch=batch, hq=hq, hkv=hkv, causal=causal)
        if kind == "block":
            c["sq"] = c["sk"] = _log_size(rng, 64, 8192)
        elif kind == "continue":
            c.update(kind="block", causal=True, sk=_log_size(rng, 1024, 65536))
            c["sq"] = _log_size(rng, 1, 1024)
        elif kind == "forward":
            c["seq"] = _log_size(rng, 1024, 131072)
        elif kind == "segments":
            c.update(shards=rng.choice((2, 4, 8)), shard=_log_size(rng, 256, 16384))
        elif kind == "steps":
            c.update(causal=False, shards=rng.choice((2, 4, 8)), shard=_log_size(rng, 256, 16384))
        elif kind == "block_backward":
            c.update(sq=_log_size(rng, 128, 8192), batch=min(batch, 2))
            c["sk"] = c["sq"]
        else:
            c.update(seq=_log_size(rng, 256, 65536), deterministic=rng.random() < 0.3)
        if work(c)["flops"] <= largest and _rows(c) * hq <= 131072 * 64:
            return c


def _rows(c):
    return c["batch"] * (c.get("seq") or c.get("sk") or c["shard"] * c["shards"])


def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda").mul_(0.5).to(torch.bfloat16)


def _attend(q, k, v, causal):
    """o (bf16) and the log-sum-exp in fp32, head by head: the forward results that a backward call is given."""
    b, sq, hq, _ = q.shape
    sk, group = k.shape[1], hq // k.shape[2]
    o, lse = torch.empty_like(q), torch.empty(b, hq, sq, device="cuda")
    hidden = None
    if causal:
        hidden = torch.ones(sq, sk, dtype=torch.bool, device="cuda").triu_(sk - sq + 1)
    for i in range(b):
        for h in range(hq):
            s = (q[i, :, h] @ k[i, :, h // group].T).float() * SCALE
            if causal:
                s.masked_fill_(hidden, -math.inf)
            lse[i, h] = torch.logsumexp(s, dim=1)
            o[i, :, h] = torch.softmax(s, dim=1).to(torch.bfloat16) @ v[i, :, h // group]
    return o, lse


def prepare(case, seed):
    c = dict(case)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, b, hq, hkv = c["kind"], c["batch"], c["hq"], c["hkv"]
    if kind in ("forward", "train"):
        c["q"] = _randn(gen, b, c["seq"], hq, D)
        c["kv"] = _randn(gen, 2, b, c["seq"], hkv, D)
        c["op"] = RingAttention((1,), b, c["seq"], hq, hkv, D, causal=c["causal"], backward=kind == "train")
        if kind == "train":
            c["dout"] = _randn(gen, b, c["seq"], hq, D)
            c["op"].deterministic_backward = c["deterministic"]
    elif kind in ("segments", "steps"):
        # the rank's own queries and every rank's K/V shard; the rank sits in the middle of the sequence
        c["rank"] = c["shards"] // 2
        c["q"] = _randn(gen, b, c["shard"], hq, D)
        c["kv"] = [_randn(gen, 2, b, c["shard"], hkv, D) for _ in range(c["shards"])]
    else:
        c["q"] = _randn(gen, b, c["sq"], hq, D)
        c["k"], c["v"] = _randn(gen, b, c["sk"], hkv, D), _randn(gen, b, c["sk"], hkv, D)
        if kind == "block_backward":
            c["dout"] = _randn(gen, b, c["sq"], hq, D)
            c["o"], c["lse"] = _attend(c["q"], c["k"], c["v"], c["causal"])
            c["dq"] = torch.empty_like(c["q"])
            c["dkv"] = torch.empty(2, b, c["sk"], hkv, D, dtype=torch.bfloat16, device="cuda")
    return c


def _order(c):
    return [(c["rank"] - t) % c["shards"] for t in range(c["shards"])]


def run(s):
    kind = s["kind"]
    if kind == "block":
        o, lse, _, _ = mb._flash_attn_forward(s["q"], s["k"], s["v"], 0.0, SCALE, s["causal"])
        return o, lse
    if kind == "forward":
        return s["op"].forward(s["q"], s["kv"])
    if kind == "train":
        o, lse = s["op"].forward(s["q"], s["kv"])
        dq, dkv = s["op"].backward(s["dout"], s["q"], s["kv"], o, lse)
        return o, lse, dq, dkv
    if kind == "segments":
        n = s["shard"]
        segs = [(s["kv"][r][0], s["kv"][r][1], r * n) for r in _order(s)]
        return mb.attn_fwd_segments(s["q"], segs, SCALE, causal=s["causal"], q_off=s["rank"] * n)
    if kind == "steps":
        # the body of a generated ring program, with the shards in place of the rotation
        out = lse = None
        for r in _order(s):
            k, v = s["kv"][r][0], s["kv"][r][1]
            params = mb.get_default_args(mb._flash_attn_forward).copy()
            params.update({"q": s["q"], "k": k, "v": v, "dropout_p": 0, "softmax_scale": SCALE, "causal": False,
                           "alibi_slopes": None, "return_softmax": False, "window_size_left": -1,
                           "window_size_right": -1})
            block_out, block_lse, _, _ = mb._flash_attn_forward(**params)
            out, lse = mb.update_out_and_lse(out, lse, block_out, block_lse)
        return out, lse
    params = mb.get_default_args(mb._flash_attn_backward).copy()
    params.update({"dout": s["dout"], "q": s["q"], "k": s["k"], "v": s["v"], "out": s["o"], "softmax_lse": s["lse"],
                   "dq": s["dq"], "dk": s["dkv"][0], "dv": s["dkv"][1], "softmax_scale": SCALE, "dropout_p": 0,
                   "causal": s["causal"], "deterministic": False, "alibi_slopes": None, "window_size_left": -1,
                   "window_size_right": -1})
    delta = mb._flash_attn_backward(**params)
    return s["dq"], s["dkv"], delta[:, :, :s["sq"]]


def _visible(case, s0, s1, q_off, sk):
    """Which of keys 0..sk-1 queries s0..s1-1 see: (number of leading keys that matter, mask of those or None)."""
    if not case["causal"]:
        return sk, None
    n = min(max(q_off + s1, 0), sk)
    pos = torch.arange(s0, s1, device="cuda")[:, None] + q_off
    return n, torch.arange(n, device="cuda")[None, :] > pos


def _exact_forward(case, q, k, v, q_off, chunk=2048):
    """o [B,S,H,D] and lse [B,H,S] of plain attention in fp64."""
    b, sq, hq, d = q.shape
    sk, group = k.shape[1], hq // k.shape[2]
    o = torch.zeros(b, sq, hq, d, dtype=torch.float64, device="cuda")
    lse = torch.full((b, hq, sq), -math.inf, dtype=torch.float64, device="cuda")
    for i in range(b):
        for h in range(hq):
            kh, vh = k[i, :, h // group].double(), v[i, :, h // group].double()
            for s0 in range(0, sq, chunk):
                s1 = min(s0 + chunk, sq)
                n, hidden = _visible(case, s0, s1, q_off, sk)
                if n == 0:
                    continue
                s = (q[i, s0:s1, h].double() @ kh[:n].T).mul_(SCALE)
                if hidden is not None:
                    s.masked_fill_(hidden, -math.inf)
                part = torch.logsumexp(s, dim=1)
                lse[i, h, s0:s1] = part
                p = s.sub_(part[:, None]).exp_().nan_to_num_(0.0)
                o[i, s0:s1, h] = p @ vh[:n]
    return o, lse


def _exact_backward(case, dout, q, k, v, o, lse, q_off, chunk=2048):
    """dq, dk, dv and rowsum(dout * o) [B,H,S] in fp64, given the forward's o and lse."""
    b, sq, hq, d = q.shape
    sk, group = k.shape[1], hq // k.shape[2]
    dq = torch.zeros(b, sq, hq, d, dtype=torch.float64, device="cuda")
    dk = torch.zeros(b, sk, hq // group, d, dtype=torch.float64, device="cuda")
    dv = torch.zeros_like(dk)
    delta = (dout.double() * o.double()).sum(-1).transpose(1, 2).contiguous()
    for i in range(b):
        for h in range(hq):
            kh, vh = k[i, :, h // group].double(), v[i, :, h // group].double()
            for s0 in range(0, sq, chunk):
                s1 = min(s0 + chunk, sq)
                n, hidden = _visible(case, s0, s1, q_off, sk)
                if n == 0:
                    continue
                qh, gh = q[i, s0:s1, h].double(), dout[i, s0:s1, h].double()
                p = (qh @ kh[:n].T).mul_(SCALE).sub_(lse[i, h, s0:s1, None].double()).exp_()
                if hidden is not None:
                    p.masked_fill_(hidden, 0.0)
                dv[i, :n, h // group] += p.T @ gh
                ds = (gh @ vh[:n].T).sub_(delta[i, h, s0:s1, None]).mul_(p).mul_(SCALE)
                dq[i, s0:s1, h] = ds @ kh[:n]
                dk[i, :n, h // group] += ds.T @ qh
    return dq, torch.stack((dk, dv)), delta


def exact(case, seed):
    """What run() returns, by plain attention in fp64 on the same inputs; None where that would take too long."""
    if work(case)["flops"] > 4.0e13:
        return None
    s, kind = prepare(case, seed), case["kind"]
    if kind in ("forward", "train"):
        o, lse = _exact_forward(case, s["q"], s["kv"][0], s["kv"][1], 0)
        if kind == "forward":
            return o, lse
        dq, dkv, _ = _exact_backward(case, s["dout"], s["q"], s["kv"][0], s["kv"][1], o, lse, 0)
        return o, lse, dq, dkv
    if kind in ("segments", "steps"):
        # the shards in sequence order: the result does not depend on the order of arrival
        kv = torch.cat(s["kv"], dim=2)
        o, lse = _exact_forward(case, s["q"], kv[0], kv[1], s["rank"] * s["shard"])
        return (o, lse.transpose(1, 2).unsqueeze(-1)) if kind == "steps" else (o, lse)
    q_off = case["sk"] - case["sq"]
    if kind == "block":
        return _exact_forward(case, s["q"], s["k"], s["v"], q_off)
    return _exact_backward(case, s["dout"], s["q"], s["k"], s["v"], s["o"], s["lse"], q_off)


def _pairs(sq, sk, q_off, causal):
    """Visible (query, key) pairs of one head; key j is visible to query i iff j <= q_off + i."""
    if not causal:
        return sq * sk
    n, first = 0, q_off + 1                    # keys that query 0 sees
    lo = max(0, 1 - first)                     # first query that sees a key
    full = min(max(sk - first, lo), sq)        # first query that sees all of them
    n += (full - lo) * (2 * first + lo + full - 1) // 2
    return n + (sq - full) * sk


def work(c):
    kind, b, hq, hkv = c["kind"], c["batch"], c["hq"], c["hkv"]
    if kind in ("forward", "train"):
        sq = sk = c["seq"]
        pairs = _pairs(sq, sk, 0, c["causal"])
    elif kind in ("segments", "steps"):
        sq, sk = c["shard"], c["shard"] * c["shards"]
        pairs = _pairs(sq, sk, c["shards"] // 2 * sq, c["causal"])
    else:
        sq, sk = c["sq"], c["sk"]
        pairs = _pairs(sq, sk, sk - sq, c["causal"])
    product = 2 * b * hq * pairs * D
    rows_q, rows_kv = b * sq * hq, b * sk * hkv
    q, kv, lse = 2 * D * rows_q, 4 * D * rows_kv, 4 * rows_q
    if kind == "train":                        # read q kv dout, write o lse dq dkv
        return {"bytes": 4 * q + 2 * kv + lse, "flops": 7 * product}
    if kind == "block_backward":               # read q kv dout o lse, write dq dkv delta
        return {"bytes": 4 * q + 2 * kv + 2 * lse, "flops": 5 * product}
    if kind == "steps":                        # the state that comes out is fp32
        return {"bytes": 3 * q + kv + lse, "flops": 2 * product}
    return {"bytes": 2 * q + kv + lse, "flops": 2 * product}


def tolerance(c):
    # Against the same attention in fp64 every bf16 output is off by 2.1e-3 to 2.4e-3 of its norm (bf16 results and bf16
    # probabilities), single values by up to 8e-2 of the root mean square; the fp32 log-sum-exp by 6e-8.
    return {"rel": 1e-2, "max": 0.3}
