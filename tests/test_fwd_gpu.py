"""Parity of the sm_100a forward kernel (through the C ABI) against the CPU oracle.

Tolerances are the ones the task states: bf16 O max-abs <= 2e-2 and LSE <= 1e-3
against fp32 attention on the same seeded inputs.
"""
import pytest
import torch

from tests.helpers import fwd_exact_and_mass, rounding_bound, seeded_qkv

pytestmark = pytest.mark.gpu

O_TOL = 2e-2
LSE_TOL = 1e-3


def _mb():
    import mercury_artifact_b200 as mb

    return mb


def _check(o, lse, ro, rl):
    o, lse = o.float().cpu(), lse.cpu()
    fin = torch.isfinite(rl)
    assert not torch.isnan(o).any()
    assert (o - ro.float()).abs().max().item() <= O_TOL
    if fin.any():
        assert (lse - rl)[fin].abs().max().item() <= LSE_TOL
    if (~fin).any():
        assert torch.equal(lse[~fin], rl[~fin])  # rows with no visible key: -inf on both sides


def _status_ok():
    from mercury_artifact_b200 import _lib

    assert _lib.status_fetch(torch.cuda.current_stream().cuda_stream) == 0


CASES = [
    # B, Sq, Sk, Hq, Hkv, causal, q_off
    (1, 256, 128, 1, 1, False, 0),
    (1, 256, 1024, 2, 2, False, 0),
    (2, 1024, 2048, 4, 4, False, 0),
    (1, 1024, 1024, 2, 2, True, 0),
    (1, 512, 1024, 2, 2, True, 512),     # bottom-right aligned causal, Sq < Sk
    (1, 1024, 512, 2, 2, True, -512),    # Sq > Sk: the first 512 rows see nothing
    (1, 300, 333, 2, 2, False, 0),       # ragged
    (2, 391, 391, 2, 2, True, 0),        # ragged + causal
    (1, 1, 1, 1, 1, False, 0),           # single query, single key
    (1, 128, 257, 1, 1, True, 129),
    (1, 512, 768, 8, 2, True, 256),      # GQA 4:1
    (2, 640, 640, 32, 8, True, 0),       # GQA, config-3 head layout
]


@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,causal,q_off", CASES)
def test_block_forward_matches_oracle(B, Sq, Sk, Hq, Hkv, causal, q_off):
    from oracle import block

    mb = _mb()
    S = max(Sq, Sk)
    q, k, v, _ = seeded_qkv(1234, B, S, Hq, Hkv, 128, device="cuda")
    q, k, v = q[:, :Sq].contiguous(), k[:, :Sk].contiguous(), v[:, :Sk].contiguous()
    scale = 128 ** -0.5
    o, lse = mb.attn_fwd_segments(q, [(k, v, 0)], scale, causal=causal, q_off=q_off)
    _status_ok()
    ro, rl = block.block_attn_fwd(q.cpu(), k.cpu(), v.cpu(), scale, causal=causal, q_off=q_off, k_off=0)
    _check(o, lse, ro, rl)


def test_drop_in_block_call_signature_and_alignment():
    """_flash_attn_forward(**params) as the generated code calls it; causal is bottom-right aligned."""
    from oracle import block

    mb = _mb()
    q, k, v, _ = seeded_qkv(7, 1, 768, 4, 4, 128, device="cuda")
    q = q[:, :256].contiguous()
    params = mb.get_default_args(mb._flash_attn_forward).copy()
    assert params["softcap"] == 0.0 and set(params) >= {"q", "k", "v", "dropout_p", "softmax_scale", "causal"}
    params.update(dict(q=q, k=k, v=v, dropout_p=0, softmax_scale=128 ** -0.5, causal=True, alibi_slopes=None,
                       return_softmax=False, window_size_left=-1, window_size_right=-1))
    outputs = mb._flash_attn_forward(**params)
    assert len(outputs) == 4
    ro, rl = block.block_attn_fwd(q.cpu(), k.cpu(), v.cpu(), 128 ** -0.5, causal=True)
    _check(outputs[0], outputs[1], ro, rl)
    assert outputs[0].dtype == q.dtype and outputs[1].dtype == torch.float32 and outputs[1].shape == (1, 4, 256)


def test_unsupported_options_raise():
    mb = _mb()
    q, k, v, _ = seeded_qkv(7, 1, 128, 1, 1, 128, device="cuda")
    with pytest.raises(NotImplementedError):
        mb._flash_attn_forward(q, k, v, 0.1, 1.0, False)
    with pytest.raises(NotImplementedError):
        mb._flash_attn_forward(q, k, v, 0.0, 1.0, False, 128, 0)
    with pytest.raises(NotImplementedError):
        mb._flash_attn_forward(q, k, v, 0.0, 1.0, False, -1, -1, 30.0)
    with pytest.raises(TypeError):
        mb.attn_fwd_segments(q.float(), [(k, v, 0)], 1.0)
    with pytest.raises(ValueError):
        mb.attn_fwd_segments(q.cpu(), [(k, v, 0)], 1.0)


def test_empty_inputs():
    mb = _mb()
    q, k, v, _ = seeded_qkv(7, 1, 256, 2, 2, 128, device="cuda")
    # no keys at all: o = 0, lse = -inf
    o, lse = mb.attn_fwd_segments(q, [(k[:, :0], v[:, :0], 0)], 1.0)
    _status_ok()
    assert (o == 0).all() and torch.isinf(lse).all() and (lse < 0).all()
    o, lse = mb.attn_fwd_segments(q, [], 1.0)
    assert (o == 0).all() and (lse == float("-inf")).all()
    # no queries: nothing to do
    o, lse = mb.attn_fwd_segments(q[:, :0], [(k, v, 0)], 1.0)
    assert o.shape[1] == 0 and lse.shape[2] == 0


def test_strided_views_of_packed_kv():
    """k = kv[0], v = kv[1] views of the packed [2,B,S,H,D] buffer, as the generated code passes them."""
    from oracle import block

    mb = _mb()
    q, k, v, _ = seeded_qkv(21, 2, 512, 4, 4, 128, device="cuda")
    kv = torch.stack([k, v]).contiguous()
    o, lse = mb.attn_fwd_segments(q, [(kv[0], kv[1], 0)], 128 ** -0.5)
    ro, rl = block.block_attn_fwd(q.cpu(), k.cpu(), v.cpu(), 128 ** -0.5)
    _check(o, lse, ro, rl)
    # sequence-sliced views (ring_divide sub-chunks)
    o2, lse2 = mb.attn_fwd_segments(q, [(kv[0][:, 128:384], kv[1][:, 128:384], 0)], 128 ** -0.5)
    ro2, rl2 = block.block_attn_fwd(q.cpu(), k[:, 128:384].cpu(), v[:, 128:384].cpu(), 128 ** -0.5)
    _check(o2, lse2, ro2, rl2)


@pytest.mark.parametrize("causal", [False, True])
def test_ring_segments_match_full_attention(causal):
    """One rank's whole ring as a single multi-segment call, in arrival order, with global positions."""
    from oracle import block
    from mercury_artifact_b200 import mesh

    mb = _mb()
    P, B, S, H = 4, 1, 2048, 4
    q, k, v, _ = seeded_qkv(99, B, S, H, H, 128, device="cuda")
    fo, fl = block.full_attention(q.cpu(), k.cpu(), v.cpu(), 128 ** -0.5, causal=causal)
    L = S // P
    for shape in [(4,), (2, 2)]:
        for r in range(P):
            order = mesh.kv_origin_schedule(r, shape)
            segs = [(k[:, o * L:(o + 1) * L], v[:, o * L:(o + 1) * L], o * L) for o in order]
            o, lse = mb.attn_fwd_segments(q[:, r * L:(r + 1) * L], segs, 128 ** -0.5, causal=causal, q_off=r * L)
            _check(o, lse, fo[:, r * L:(r + 1) * L], fl[:, :, r * L:(r + 1) * L])
    _status_ok()


@pytest.mark.parametrize("causal", [False, True])
def test_growing_scores_force_the_output_rescale(causal):
    """Keys whose scores grow from tile to tile: the running row max rises by far more than the lazy-rescale
    threshold (2^8 in the exponent), so the accumulated output is rescaled in tensor memory several times; the
    last segment repeats the growth across a segment boundary."""
    from oracle import block

    mb = _mb()
    B, S, H = 1, 1536, 2
    q, k, v, _ = seeded_qkv(5, B, S, H, H, 128, device="cuda")
    ramp = torch.linspace(1.0, 24.0, S, device="cuda").view(1, S, 1, 1)   # |score| grows ~24x along the keys
    k = (k.float() * ramp).bfloat16()
    fo, fl = block.full_attention(q.cpu(), k.cpu(), v.cpu(), 128 ** -0.5, causal=causal)
    o, lse = mb.attn_fwd_segments(q, [(k, v, 0)], 128 ** -0.5, causal=causal)
    _check(o, lse, fo, fl)
    segs = [(k[:, :640], v[:, :640], 0), (k[:, 640:], v[:, 640:], 640)]
    o, lse = mb.attn_fwd_segments(q, segs, 128 ** -0.5, causal=causal)
    _check(o, lse, fo, fl)
    _status_ok()


@pytest.mark.parametrize("causal,chunks", [(True, 4), (True, 16), (False, 4), (True, 3)])
def test_host_buffer_forward_matches_oracle(causal, chunks):
    """forward_host(): pinned host tensors in and out, sequence chunks pipelined over PCIe (chunks=3 does not
    divide into 128-row pieces and takes the plain copy-in / forward / copy-out path)."""
    from oracle import block
    from mercury_artifact_b200.ring import RingAttention

    B, S, H = 1, 2048, 4
    q, k, v, _ = seeded_qkv(7, B, S, H, H, 128, device="cpu")
    fo, fl = block.full_attention(q, k, v, 128 ** -0.5, causal=causal)
    q_host = q.contiguous().pin_memory()
    kv_host = torch.stack([k, v]).contiguous().pin_memory()
    o_host = torch.empty_like(q_host).pin_memory()
    lse_host = torch.empty((B, H, S), dtype=torch.float32).pin_memory()
    op = RingAttention((1,), B, S, H, H, 128, causal=causal)
    for _ in range(2):  # twice: the second call reuses the device buffers and streams
        o_host.zero_()
        lse_host.zero_()
        op.forward_host(q_host, kv_host, o_host, lse_host, chunks=chunks)
        _check(o_host, lse_host, fo, fl)
    _status_ok()


def test_full_size_properties_config2():
    """The headline benchmark shape (bf16 B1 S32768 H32 D128 causal): size-independent properties.

    * splitting K/V into segments at tile boundaries does not change a single bit;
    * query row 0 of a causal run attends to key 0 only: o[0] == v[0], lse[0] == scale * q0.k0;
    * merging the two half-sequence partial results reproduces the one-pass result.
    """
    mb = _mb()
    B, S, H = 1, 32768, 32
    q, k, v, _ = seeded_qkv(1234, B, S, H, H, 128, device="cuda")
    scale = 128 ** -0.5
    o1, l1 = mb.attn_fwd_segments(q, [(k, v, 0)], scale, causal=True)
    h = S // 2
    o2, l2 = mb.attn_fwd_segments(q, [(k[:, :h], v[:, :h], 0), (k[:, h:], v[:, h:], h)], scale, causal=True)
    _status_ok()
    assert torch.equal(o1, o2) and torch.equal(l1, l2)
    assert torch.equal(o1[:, 0], v[:, 0])
    want = (q[:, 0].float() * k[:, 0].float()).sum(-1) * scale
    assert (l1[:, :, 0] - want).abs().max().item() <= LSE_TOL
    # partials over disjoint key halves, merged by the drop-in merge
    pa, la = mb.attn_fwd_segments(q, [(k[:, :h], v[:, :h], 0)], scale, causal=True)
    pb, lb = mb.attn_fwd_segments(q[:, h:], [(k[:, h:], v[:, h:], h)], scale, causal=True, q_off=h)
    out, lse = mb.update_out_and_lse(None, None, pa[:, h:], la[:, :, h:].contiguous())
    out, lse = mb.update_out_and_lse(out, lse, pb, lb)
    assert (out - o1[:, h:].float()).abs().max().item() <= O_TOL
    assert (lse.squeeze(-1).transpose(1, 2) - l1[:, :, h:]).abs().max().item() <= LSE_TOL
    assert torch.equal(pa[:, :h], o1[:, :h])


@pytest.mark.gpu
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("one_launch", [False, True])
def test_carried_state_chain_equals_one_job_bitwise(causal, one_launch):
    """A query shard processed as a chain of jobs, one per K/V shard, each continuing the online-softmax
    state the previous one stored (mb_fwd_job.state_*), gives the bits of one job over all the shards:
    as separate launches of one stream, and as ONE launch whose jobs hand over through chain words.
    Ragged sizes, GQA, a shard that the early query rows cannot see (their state passes through), and a
    first shard that late-positioned keys make invisible to every row of some tiles."""
    import mercury_artifact_b200 as mb
    from mercury_artifact_b200 import _lib
    from mercury_artifact_b200.attention import attn_fwd_multi
    from tests.helpers import seeded_qkv

    dev = torch.device("cuda", 0)
    B, Sq, Sk, H, hkv, D = 2, 1000, 1400, 4, 2, 128
    q, _, _, _ = seeded_qkv(5, B, Sq, H, hkv, D, device="cuda")
    _, k, v, _ = seeded_qkv(6, B, Sk, H, hkv, D, device="cuda")
    scale = D ** -0.5
    q_off = 300
    # K/V shards in "arrival" order: the middle one first (keys 500..899 are invisible to rows < 200 when
    # causal), then the head, then the tail (1 000..1 399: invisible to most rows, ragged)
    cuts = [(500, 900), (0, 500), (900, 1400)]
    segs = [(k[:, a:b], v[:, a:b], a) for a, b in cuts]
    ref_o, ref_l = mb.attn_fwd_segments(q, segs, scale, causal=causal, q_off=q_off)

    o = torch.full_like(q, 7.0)
    lse = torch.full((B, H, Sq), 7.0, device=dev)
    st_o = torch.full((B, H, Sq, D), float("nan"), device=dev)
    st_ml = torch.full((B, H, Sq, 2), float("nan"), device=dev)
    n_pairs = (Sq + 255) // 256
    chain = torch.zeros(B, H, n_pairs, dtype=torch.int32, device=dev)
    jobs = []
    for t in range(len(segs)):
        j = {"q": q, "q_off": q_off, "seg_mask": 1 << t, "state": (st_o, st_ml),
             "state_in": t > 0, "state_out": t < len(segs) - 1}
        if t == len(segs) - 1:
            j["out_raw"] = (o.data_ptr(), o.stride(0), o.stride(1), o.stride(2))
            j["lse_raw"] = (lse.data_ptr(), lse.stride(0), lse.stride(1))
        if one_launch:
            j["chain"] = (chain.data_ptr(), t, t + 1)
        jobs.append(j)
    if one_launch:
        attn_fwd_multi(jobs, segs, scale, causal, B, H, hkv, D, dev)
    else:
        for j in jobs:
            attn_fwd_multi([j], segs, scale, causal, B, H, hkv, D, dev)
    assert _lib.status_fetch(torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(o, ref_o)
    assert torch.equal(lse, ref_l)
    if one_launch:
        assert chain.unique().tolist() == [len(segs) - 1]


@pytest.mark.gpu
def test_carried_state_is_the_unnormalised_accumulator():
    """What a state_out job stores: rows o * l with l the sum of exp(scale * (s - m)) and m the stored
    maximum, so that o = state_o / l and lse = scale * m + ln(l) reproduce the one-job result; rows without
    a visible key store (0, -inf, 0).  Two chains in one launch (two query shards) do not disturb each other."""
    import mercury_artifact_b200 as mb
    from mercury_artifact_b200 import _lib
    from mercury_artifact_b200.attention import attn_fwd_multi
    from tests.helpers import seeded_qkv

    dev = torch.device("cuda", 0)
    B, S, H, D = 1, 512, 2, 128
    q, k, v, _ = seeded_qkv(9, B, S, H, H, D, device="cuda")
    scale = D ** -0.5
    segs = [(k[:, 256:], v[:, 256:], 256), (k[:, :256], v[:, :256], 0)]
    ref_o, ref_l = mb.attn_fwd_segments(q, segs, scale, causal=True, q_off=0)
    halves = [slice(0, 256), slice(256, 512)]
    o = torch.zeros_like(q)
    lse = torch.zeros(B, H, S, device=dev)
    states = [(torch.zeros(B, H, 256, D, device=dev), torch.zeros(B, H, 256, 2, device=dev)) for _ in halves]
    chain = torch.zeros(2, B, H, 1, dtype=torch.int32, device=dev)
    jobs = []
    for t in range(2):                      # shard-major order: both chains' first jobs, then their second ones
        for c, rows in enumerate(halves):
            j = {"q": q[:, rows], "q_off": rows.start, "seg_mask": 1 << t, "state": states[c],
                 "state_in": t == 1, "state_out": t == 0, "chain": (chain[c].data_ptr(), t, t + 1)}
            if t == 1:
                j["out_raw"] = (o[:, rows].data_ptr(), o.stride(0), o.stride(1), o.stride(2))
                j["lse_raw"] = (lse[:, :, rows].data_ptr(), lse.stride(0), lse.stride(1))
            jobs.append(j)
    attn_fwd_multi(jobs[:2], segs, scale, True, B, H, H, D, dev)      # first jobs alone: look at the state
    torch.cuda.synchronize()
    so, sml = states[0]                    # rows 0..255 see nothing of keys 256..511
    assert so.abs().max().item() == 0 and torch.isneginf(sml[..., 0]).all() and (sml[..., 1] == 0).all()
    so, sml = states[1]                    # rows 256..511 against keys 256..511, causal
    po, pl = mb.attn_fwd_segments(q[:, 256:], segs[:1], scale, causal=True, q_off=256)
    m, l = sml[..., 0], sml[..., 1]
    assert (l > 0).all()
    assert ((so / l[..., None]).transpose(1, 2) - po.float()).abs().max().item() <= 2e-2
    assert (m * scale + l.log() - pl).abs().max().item() <= 1e-3
    chain.zero_()
    attn_fwd_multi(jobs, segs, scale, True, B, H, H, D, dev)
    assert _lib.status_fetch(torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(o, ref_o) and torch.equal(lse, ref_l)


@pytest.mark.gpu
@pytest.mark.parametrize("causal", [False, True])
def test_eight_chains_of_one_launch_like_one_rank_of_eight(causal):
    """The launch one rank of an 8-rank heads schedule issues, with all data local: 8 query chunks x 8 K/V shards
    in an arrival order that starts in the middle, 36 jobs (causal: 24) that share 8 query tensor maps, one
    state chain per chunk -- the first job of a chunk takes every shard that arrived before its queries did.
    Bit-identical to one job per chunk over the same shard order."""
    import mercury_artifact_b200 as mb
    from mercury_artifact_b200 import _lib
    from mercury_artifact_b200.attention import attn_fwd_multi
    from tests.helpers import seeded_qkv

    dev = torch.device("cuda", 0)
    P, B, L, H, hkv, D = 8, 1, 512, 2, 1, 128
    S = P * L
    q, k, v, _ = seeded_qkv(77, B, S, H, hkv, D, device="cuda")
    scale = D ** -0.5
    me = 5
    order = [me] + [(me - t) % P for t in range(1, P)]
    segs = [(k[:, s * L:(s + 1) * L], v[:, s * L:(s + 1) * L], s * L) for s in order]
    o = torch.zeros_like(q)
    lse = torch.zeros(B, H, S, device=dev)
    states = [(torch.empty(B, H, L, D, device=dev), torch.empty(B, H, L, 2, device=dev),
               torch.zeros(B, H, L // 256, dtype=torch.int32, device=dev)) for _ in range(P)]
    plan = []
    for t in range(P):
        for n in range(t + 1):
            j = order[n]
            shards = range(t + 1) if n == t else (t,)
            mask = sum(1 << i for i in shards if (not causal) or order[i] <= j)
            if mask:
                plan.append((n, mask))
    count = [sum(1 for n, _ in plan if n == c) for c in range(P)]
    seen = [0] * P
    jobs = []
    for n, mask in plan:
        j = order[n]
        p, last = seen[n], seen[n] == count[n] - 1
        seen[n] += 1
        jb = {"q": q[:, j * L:(j + 1) * L], "q_off": j * L, "seg_mask": mask}
        if count[n] > 1:
            jb.update(state=states[n][:2], state_in=p > 0, state_out=not last, chain=(states[n][2].data_ptr(), p, p + 1))
        if last:
            jb["out_raw"] = (o[:, j * L:].data_ptr(), o.stride(0), o.stride(1), o.stride(2))
            jb["lse_raw"] = (lse[:, :, j * L:].data_ptr(), lse.stride(0), lse.stride(1))
        jobs.append(jb)
    assert len(jobs) == (24 if causal else 36)      # more than one launch used to take
    attn_fwd_multi(jobs, segs, scale, causal, B, H, hkv, D, dev)
    assert _lib.status_fetch(torch.cuda.current_stream().cuda_stream) == 0
    for j in range(P):
        ro, rl = mb.attn_fwd_segments(q[:, j * L:(j + 1) * L], segs, scale, causal=causal, q_off=j * L)
        assert torch.equal(o[:, j * L:(j + 1) * L], ro), j
        assert torch.equal(lse[:, :, j * L:(j + 1) * L], rl), j


SPLIT_CASES = [
    # B, Sq, Sk, Hq, Hkv, causal, q_off, K/V shards, does the launch split items over their keys
    (1, 1, 3001, 8, 2, False, 0, 1, True),        # one query, four heads to a tile
    (1, 100, 4096, 8, 2, True, 3996, 1, True),    # shares of a causal item; heads packed
    (2, 77, 2500, 16, 4, True, 2423, 1, True),    # ragged everywhere
    (1, 300, 2049, 4, 4, False, 0, 1, True),      # more queries than one item, last key tile of one key
    (1, 700, 1600, 8, 8, True, 0, 1, True),       # early rows: shares without a visible key
    (1, 1300, 900, 2, 2, True, -300, 1, True),    # rows without any visible key in every share
    (1, 33, 1500, 6, 2, False, 0, 1, True),       # a group that does not divide a tile: heads apart
    (1, 65, 300, 128, 1, True, 235, 1, False),    # the largest group that fits a tile; too few keys to split
    (1, 65, 900, 128, 1, True, 835, 1, True),     # the same with enough
    (3, 6390, 1400, 2, 2, False, 0, 1, True),     # 150 items: the last two split, the first 148 whole
    (3, 6390, 1400, 2, 2, False, 0, 3, True),     # the same over three shards
    (2, 300, 1400, 4, 2, True, 1100, 3, False),   # several shards, less than a wave: whole
]


@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,causal,q_off,shards,splits", SPLIT_CASES)
def test_items_split_over_their_keys_match_oracle(B, Sq, Sk, Hq, Hkv, causal, q_off, shards, splits, monkeypatch):
    """Launches that share a work item between CTAs (and merge the shares), and tiles that hold the rows of all
    heads of a group.  Every element keeps the bound that the kernel's roundings give (the shares are merged in fp32):
    the outputs are small, 0.01 in the mean of squares, and a share that is lost moves them by less than O_TOL."""
    import mercury_artifact_b200 as mb
    from mercury_artifact_b200 import _lib
    from oracle import block

    q, k, v, _ = seeded_qkv(11, B, max(Sq, Sk), Hq, Hkv, 128)
    q, k, v = q[:, :Sq], k[:, :Sk], v[:, :Sk]
    scale = 128 ** -0.5
    need = []
    real_lib = _lib.lib

    class Lib:
        def __getattr__(self, name):
            return getattr(real_lib, name)

        def mb_attn_fwd_workspace(self, args):
            need.append(real_lib.mb_attn_fwd_workspace(args))
            return need[-1]

    monkeypatch.setattr(_lib, "lib", Lib())
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    cut = [Sk * i // shards for i in range(shards + 1)]
    segs = [(kd[:, a:b], vd[:, a:b], a) for a, b in zip(cut[:-1], cut[1:])]
    o, lse = mb.attn_fwd_segments(qd, segs, scale, causal=causal, q_off=q_off)
    monkeypatch.undo()
    _status_ok()
    assert (need[0] > 0) == splits
    # the long case: rows of whole and of split items
    for rows in [slice(0, Sq)] if Sq < 5000 else [slice(Sq - 700, Sq), slice(0, 300)]:
        off = q_off + rows.start
        ro, rl = block.block_attn_fwd(q[:, rows], k, v, scale, causal=causal, q_off=off)
        _check(o[:, rows], lse[:, :, rows], ro, rl)
        exact, mass = fwd_exact_and_mass(q[:, rows], k, v, scale, causal, off)
        assert ((o[:, rows].float().cpu() - exact).abs() <= rounding_bound(mass, exact)).all()
    # all rows against the call without a workspace, which does not split: the roundings of both
    ow, lw = torch.empty_like(qd), torch.empty_like(lse)
    raw = dict(out_raw=(ow.data_ptr(), *ow.stride()[:3]), lse_raw=(lw.data_ptr(), *lw.stride()[:2]))
    mb.attn_fwd_segments(qd, segs, scale, causal=causal, q_off=q_off, **raw)
    mass = torch.empty_like(qd)
    raw["out_raw"] = (mass.data_ptr(), *mass.stride()[:3])
    va = torch.empty_strided(vd.shape, vd.stride(), dtype=vd.dtype, device="cuda").copy_(vd.abs())
    mb.attn_fwd_segments(qd, [(kd[:, a:b], va[:, a:b], a) for a, b in zip(cut[:-1], cut[1:])], scale, causal=causal,
                         q_off=q_off, **raw)
    _status_ok()
    ow, mass = ow.float(), mass.float() * (1 + 2.0 ** -7)   # (the mass is itself rounded twice)
    assert ((o.float() - ow).abs() <= 2 * rounding_bound(mass, ow)).all()
    seen = ~lw.isneginf()
    assert torch.equal(lse.isneginf(), ~seen) and (lse - lw)[seen].abs().max().item() <= 1e-5


def test_split_calls_and_merges_under_graph_capture():
    """Block calls that split (workspace, merge launch), overlapped launches and the running merge, captured into a
    graph and replayed on other inputs: the bits of the same calls outside."""
    import mercury_artifact_b200 as mb

    B, Sq, Sk, H, hkv, D = 1, 100, 4096, 8, 2, 128
    scale = D ** -0.5
    sets = [seeded_qkv(s, B, Sk, H, hkv, D, device="cuda")[:3] for s in (41, 51)]
    q, k, v = sets[0][0][:, :Sq].contiguous(), sets[0][1].clone(), sets[0][2].clone()

    def step():
        out = lse = None
        for half in (slice(0, Sk // 2), slice(Sk // 2, Sk)):
            o, l, _, _ = mb._flash_attn_forward(q, k[:, half], v[:, half], 0.0, scale, False)
            out, lse = mb.update_out_and_lse(out, lse, o, l)
        return out, lse

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out, lse = step()
    for q2, k2, v2 in reversed(sets):
        q.copy_(q2[:, :Sq])
        k.copy_(k2)
        v.copy_(v2)
        for _ in range(3):
            graph.replay()
        ro, rl = step()
        assert torch.equal(out, ro) and torch.equal(lse, rl)
    _status_ok()


@pytest.mark.parametrize("B,Sq,H,hkv,causal,q_off,splits", [
    (3, 6390, 2, 2, False, 0, True),     # 150 items, of which attn_fwd_segments splits the last two
    (2, 300, 4, 2, True, 1100, False),   # one wave: whole, heads apart
    (1, 100, 8, 2, True, 1300, False),
    (16, 300, 8, 2, True, 1100, False),  # 256 pairs with the heads of a group apart: packed (attn_fwd_multi does not)
    (1, 180, 8, 2, True, 2500, False),   # one wave, both tiles of the longest pair and more than 16 key tiles: packed
])
def test_ways_that_never_split_keep_each_others_bits(B, Sq, H, hkv, causal, q_off, splits):
    """Over three shards, mb_attn_fwd (no workspace), one job of attn_fwd_multi and a chain of three jobs agree bit for
    bit at every size, as mercury_b200.h says.  A call that splits agrees with them bit for bit in its whole
    items and to the rounding of bf16 probabilities in the others."""
    import mercury_artifact_b200 as mb
    from mercury_artifact_b200.attention import attn_fwd_multi

    Sk, D = max(1400, Sq + q_off if causal else 0), 128
    dev = torch.device("cuda", 0)
    q, _, _, _ = seeded_qkv(11, B, Sq, H, hkv, D, device="cuda")
    _, k, v, _ = seeded_qkv(12, B, Sk, H, hkv, D, device="cuda")
    scale = D ** -0.5
    cut = [Sk * i // 3 for i in range(4)]
    segs = [(k[:, a:b], v[:, a:b], a) for a, b in zip(cut[:-1], cut[1:])]

    def multi(masks):
        o, lse = torch.empty_like(q), torch.empty(B, H, Sq, device=dev)
        state = (torch.empty(B, H, Sq, D, device=dev), torch.empty(B, H, Sq, 2, device=dev))
        chain = torch.zeros(B, H, (Sq + 255) // 256, dtype=torch.int32, device=dev)
        jobs = [{"q": q, "q_off": q_off, "seg_mask": m} for m in masks]
        for t, j in enumerate(jobs):
            if len(jobs) > 1:
                j.update(state=state, state_in=t > 0, state_out=t < len(jobs) - 1, chain=(chain.data_ptr(), t, t + 1))
        jobs[-1]["out_raw"] = (o.data_ptr(), *o.stride()[:3])
        jobs[-1]["lse_raw"] = (lse.data_ptr(), *lse.stride()[:2])
        attn_fwd_multi(jobs, segs, scale, causal, B, H, hkv, D, dev)
        return o, lse

    o1, l1 = multi([7])
    o3, l3 = multi([1, 2, 4])
    ow, lw = torch.empty_like(q), torch.empty(B, H, Sq, device=dev)   # raw results: the wrapper gives no workspace
    mb.attn_fwd_segments(q, segs, scale, causal=causal, q_off=q_off, out_raw=(ow.data_ptr(), *ow.stride()[:3]),
                         lse_raw=(lw.data_ptr(), *lw.stride()[:2]))
    os_, ls = mb.attn_fwd_segments(q, segs, scale, causal=causal, q_off=q_off)
    _status_ok()
    for o, lse in ((o3, l3), (ow, lw)):
        assert torch.equal(o, o1) and torch.equal(lse, l1)
    if not splits:
        assert torch.equal(os_, o1) and torch.equal(ls, l1)
        return
    differ = (os_ != o1).any(-1)
    whole = torch.ones_like(differ)
    whole[2, 23 * 256:, 1] = False            # items 148 and 149: the last two pairs of tiles of the last head
    assert not (differ & whole).any() and differ.any()
    err = (os_.float() - o1.float())[~whole].norm() / o1.float()[~whole].norm()
    assert err.item() <= 1e-2
    assert (ls - l1).abs().max().item() <= LSE_TOL


@pytest.mark.parametrize("Sq,splits", [(600, True), (13900, False)])
def test_items_in_uneven_head_blocks(Sq, splits, monkeypatch):
    """Causal launches take the items of several heads together, as many heads as have their K/V in 64 MiB: 11 heads of
    16 384 keys go as 6 + 5, with split items (and their merge) and without.  A launch with an arrival flag
    (raised beforehand) goes head by head and whole, and gives the same bits where nothing was split."""
    import mercury_artifact_b200 as mb
    from mercury_artifact_b200 import _lib

    Sk, H, D = 16384, 11, 128
    scale = D ** -0.5
    q_off = Sk - Sq - 50
    q, _, _, _ = seeded_qkv(81, 1, Sq, H, H, D, device="cuda")
    _, k, v, _ = seeded_qkv(82, 1, Sk, H, H, D, device="cuda")
    real, need = _lib.lib, []

    class Lib:
        def __getattr__(self, name):
            return getattr(real, name)

        def mb_attn_fwd_workspace(self, args):
            need.append(real.mb_attn_fwd_workspace(args))
            return need[-1]

    monkeypatch.setattr(_lib, "lib", Lib())
    o, lse = mb.attn_fwd_segments(q, [(k, v, 0)], scale, causal=True, q_off=q_off)
    monkeypatch.undo()
    assert (need[0] > 0) == splits
    flag = torch.ones(1, dtype=torch.int32, device="cuda")
    seg = (k, v, 0, flag.data_ptr(), 1)
    ow, lw = mb.attn_fwd_segments(q, [seg], scale, causal=True, q_off=q_off)
    mass, _ = mb.attn_fwd_segments(q, [(k, v.abs(), *seg[2:])], scale, causal=True, q_off=q_off)
    _status_ok()
    if not splits:
        assert torch.equal(o, ow) and torch.equal(lse, lw)
    ow, mass = ow.float(), mass.float() * (1 + 2.0 ** -7)
    assert ((o.float() - ow).abs() <= 2 * rounding_bound(mass, ow)).all()
    assert (lse - lw).abs().max().item() <= 1e-5


@pytest.mark.parametrize("rows,heads,splits", [(4352, 8, True), (4864, 8, False), (5000, 8, False), (6144, 8, False),
                                               (2048, 8, True), (9728, 4, True)])
def test_causal_launches_split_where_it_is_faster(rows, heads, splits):
    """What mb_attn_fwd_workspace asks for around one wave of causal items (148 SMs): 4 864 to 6 144 rows with 8 heads were
    split and slower for it, 9 728 rows with 4 heads have few long items; 2 048 rows take 2 shares, which fit a wave."""
    from mercury_artifact_b200 import _lib

    a = _lib.AttnFwdArgs()
    a.batch, a.sq, a.hq, a.hkv, a.head_dim, a.causal, a.softmax_scale, a.nseg = 1, rows, heads, heads, 128, 1, 0.1, 1
    a.seg[0].sk = rows
    slots = _lib.lib.mb_attn_fwd_workspace(a) // (256 * (128 * 4 + 8))
    items = (rows + 255) // 256 * heads
    assert slots == (items * 2 if splits else 0)



@pytest.mark.parametrize("heads,rows,keys", [(4, 5120, 1024), (4, 5120, 4096), (4, 2304, 4096), (4, 8960, 4096)])
def test_launches_that_overlap_and_that_do_not_read_what_the_one_before_wrote(heads, rows, keys):
    """Calls of one wave back to back, on both sides of the rule for overlapped launches (80 pairs of 8 and of 32 steps, 36
    and 140 of 32), each on the output of the one before: the bits of the same calls with the device idle in between."""
    import mercury_artifact_b200 as mb

    q, _, _, _ = seeded_qkv(91, 1, rows, heads, heads, 128, device="cuda")
    _, k, v, _ = seeded_qkv(92, 1, keys, heads, heads, 128, device="cuda")
    half = keys // 2
    segs = [(k[:, :half], v[:, :half], 0), (k[:, half:], v[:, half:], half)]

    def chain(pause):
        x = q
        for _ in range(5):
            x, lse = mb.attn_fwd_segments(x * 30.0, segs, 128 ** -0.5)
            if pause:
                torch.cuda.synchronize()
        return x, lse

    a, b = chain(False), chain(True)
    _status_ok()
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
