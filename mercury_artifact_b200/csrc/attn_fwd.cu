// Forward attention over a list of K/V segments for sm_100a.
//
// One CTA owns two 128-row query tiles of one (batch, query-head) and streams
// every K/V tile of every segment through them, keeping the online-softmax
// state (row max, row sum, fp32 output accumulator) on chip for the whole list.
// A "segment" is one sequence shard of K and V: the per-step block of the ring
// schedule is a one-segment call, and the whole ring (or double ring) for one
// rank is an nseg-segment call whose segment order is the rank's arrival order.
// Because the running state never leaves the SM, the per-step out/LSE merge of
// the generated ring loop (utils/flash_attn_dsl.py:31-71 in the reference)
// disappears from the fused path.
//
// Roles inside the CTA (384 threads, three warpgroups):
//   warps 0-3  softmax + epilogue for query tile 0 (one thread per row)
//   warps 4-7  softmax + epilogue for query tile 1
//   warp  8    tcgen05.mma issuer for the Q.K^T products of both query tiles, tensor-memory owner
//   warp  9    TMA loader (lane 0)
//   warp 10    tcgen05.mma issuer for the P.V products of both query tiles
//   warp 11    idle; the auxiliary warpgroup's registers go to the softmax warps (setmaxnreg)
//
// Tensor memory (512 columns): S | P0 | P1 | O0 | O1 = 128 + 64 + 64 + 128 + 128.  There is ONE
// fp32 score region, used by the two query tiles in turn: a softmax thread copies its whole score
// row into registers as soon as the tile is complete and hands the region on, so the next Q.K^T
// product (of the other query tile) starts while this tile is still in its exponentials.  The bf16
// probabilities have a region of their own per query tile, so that the next score tile of a query
// tile does not have to wait for its P.V product either.  What remains serial is the hand-over of
// the score region: copy-out -> issuing warp wakes -> 8 MMAs -> tensor-pipe latency -> softmax warp
// wakes, about 1 100-1 300 cycles per use, two uses per K/V tile.
//
// K/V tiles are loaded in the order K0 K1 V0 K2 V1 K3 V2 ...: the score product of K/V tile g+1 is
// issued before the P.V product of tile g needs its V tile.
//
// A launch may carry several "jobs": query shards with their own output pointers, sharing the segment
// list.  blockIdx.x runs through the query-tile pairs of job 0, then of job 1, ...  A job can name an
// arrival flag for its queries (they may still be in flight from another GPU) and a completion flag,
// which the job's last CTA raises with a release store at system scope once every row of the job has
// been stored -- the rows, and the flag, may live in another GPU's memory.
//
// A single job without flags may be cut differently (see plan_pack and plan_split): a tile then holds the rows of
// all heads of a group, and an item's K/V tiles are shared between several CTAs, whose states
// fwd_split_merge_kernel merges.
#include <climits>

#include "attn_fwd_common.cuh"

namespace mb {

// Position in the CTA's list of K/V tiles: every tile of every segment that at least one of the two
// query tiles takes part in, in segment order.
struct TileIter {
  int s, jt;
};
__device__ __forceinline__ int seg_tiles(const FwdSmem* ctl, int s) {
  return max(ctl->n_tiles[0][s], ctl->n_tiles[1][s]);
}
// First tile of a segment that this CTA has (kCut: the launch splits items or packs heads).
template <bool kCut>
__device__ __forceinline__ int seg_first(const FwdSmem* ctl, int s) {
  if constexpr (kCut) return ctl->t_lo[s];
  return 0;
}
template <bool kCut>
__device__ __forceinline__ TileIter iter_first(const FwdSmem* ctl, int nseg) {
  TileIter it{0, 0};
  while (it.s < nseg && seg_tiles(ctl, it.s) <= seg_first<kCut>(ctl, it.s)) ++it.s;
  if (it.s < nseg) it.jt = seg_first<kCut>(ctl, it.s);
  return it;
}
template <bool kCut>
__device__ __forceinline__ void iter_next(const FwdSmem* ctl, int nseg, TileIter& it) {
  if (++it.jt >= seg_tiles(ctl, it.s)) {
    ++it.s;
    while (it.s < nseg && seg_tiles(ctl, it.s) <= seg_first<kCut>(ctl, it.s)) ++it.s;
    it.jt = it.s < nseg ? seg_first<kCut>(ctl, it.s) : 0;
  }
}

// Query tile pair, head and batch entry of a job's work item.  (batch entry, head) pairs are taken in blocks of
// `hb`; inside a block the pairs come row by row, heavier (later) query rows first when causal, and the heads
// of one row one after the other.  hb = 1 is head by head.
struct ItemCoords {
  int pair, h, b;
};
__device__ __forceinline__ ItemCoords item_coords(int item, int n_pairs, int hb, int B, int Hq, int causal) {
  const int blk = item / (hb * n_pairs), rem = item - blk * hb * n_pairs;
  const int n = min(hb, B * Hq - blk * hb);  // heads of this block
  const int pidx = rem / n, bh = blk * hb + rem % n;
  return ItemCoords{causal ? n_pairs - 1 - pidx : pidx, bh % Hq, bh / Hq};
}

// Register budgets.  setmaxnreg can only redistribute the registers the CTA was launched with
// (threads x launch budget); an increase beyond that pool would block forever, hence the check.
#define MB_FWD_LAUNCH_REGS 160
#define MB_FWD_SOFTMAX_REGS 216
#define MB_FWD_AUX_REGS 48
#define MB_STR2(x) #x
#define MB_STR(x) MB_STR2(x)
static_assert(8 * 32 * MB_FWD_SOFTMAX_REGS + 4 * 32 * MB_FWD_AUX_REGS <= kFwdThreads * MB_FWD_LAUNCH_REGS,
              "setmaxnreg budgets exceed the registers the CTA is launched with");

// 160 registers/thread at launch (not the 168 that 384 threads would allow): the few warps' worth
// left free on the SM let the transfer stream's one-thread flag kernels start beside a resident CTA.
//
// kCut: the launch splits items over their keys or packs the heads of a group.  The others, every launch with several jobs
// among them, take an instantiation without what that needs, which short items feel (one instantiation / two): 8 x 256 x
// 256, 32 heads 23.5 / 22.7 us, 16 x 256 x 256 49.3 / 47.7, 4 x 512 x 512 29.2 / 28.8; 8 192 x 8 192 the same.
template <bool kCut>
__global__ void __maxnreg__(MB_FWD_LAUNCH_REGS)
attn_fwd_kernel(const __grid_constant__ FwdMaps maps, const __grid_constant__ FwdArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + 2 * kTileBytes;
  FwdSmem* ctl = reinterpret_cast<FwdSmem*>(smem + 2 * kTileBytes + kFwdStages * kTileBytes);
  volatile int* abort_word = &ctl->abort_word;

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int pack_shift = kCut ? a.pack_shift : 0;

  if (a.overlap) grid_dependents_launch();
  // Which job this CTA belongs to; within a job the heavier (later) query rows come first when causal.
  if (tid == 0) {
    int jid = 0;
    while (jid + 1 < a.njobs && (int)blockIdx.x >= a.job[jid + 1].x_begin) ++jid;
    ctl->jid = jid;
    ctl->job = a.job[jid];
    // CTAs are dispatched in grid order: job by job, inside a job in the order of item_coords (the CTAs
    // running at one time share a few heads' K/V through L2).
    int local = (int)blockIdx.x - a.job[jid].x_begin;
    if constexpr (kCut) {
      ctl->slot = -1;
      ctl->part = 0;
      if (local >= a.split_begin) {
        ctl->slot = local - a.split_begin;
        ctl->part = ctl->slot % a.nsplit;
        local = a.split_begin + ctl->slot / a.nsplit;
      }
    }
    const ItemCoords it = item_coords(local, a.job[jid].n_pairs, a.head_block, a.B, a.Hq >> pack_shift, a.causal);
    ctl->pair = it.pair;
    ctl->h = it.h << pack_shift;
    ctl->b = it.b;
  }
  __syncthreads();
  const FwdJob& J = ctl->job;
  // (pair, head, batch entry) stay in shared memory: the roles read them where they need them, so that
  // they occupy no registers across the softmax loop
  const int q0 = ctl->pair * 2 * kBM;

  if (tid == 0) {
    mbar_init(&ctl->q_full, 1);
    for (int s = 0; s < kFwdStages; ++s) {
      mbar_init(&ctl->kv_full[s], 1);
      mbar_init(&ctl->kv_empty[s], 1);  // released by the one warp that consumes the stage
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ctl->s_full[i], 1);
      mbar_init(&ctl->p_full[i][0], 128);
      mbar_init(&ctl->p_full[i][1], 128);
      mbar_init(&ctl->o_full[i], 1);
    }
    mbar_init(&ctl->s_free, 4);
    mbar_init(&ctl->drain, 2);
    ctl->abort_word = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  // K/V tiles of each segment that each of the two query tiles takes part in: one lane per segment
  // (computed by one thread this was ~4 000 cycles of a CTA's prologue at 32 segments)
  static_assert(MB_MAX_SEGMENTS == 32, "one lane of warp 0 per segment");
  if (warp == 0) {
    int n[2] = {0, 0};
    if (lane < a.nseg && ((J.seg_mask >> lane) & 1u)) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
        n[i] = visible_tiles(q0 + i * kBM, J.Sq, pack_shift, J.q_off, a.causal, a.seg_sk[lane], a.seg_koff[lane]);
    }
    int lo = 0;
    if (kCut && ctl->slot >= 0) {
      // This CTA's share of the item's walk over all its K/V tiles: an equal part, cut at whole tiles.
      const int mine = max(n[0], n[1]);
      int incl = mine;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += up;
      }
      const long long all = __shfl_sync(0xffffffffu, incl, 31);
      const int before = incl - mine;
      const int first = (int)(all * ctl->part / a.nsplit), last = (int)(all * (ctl->part + 1) / a.nsplit);
      lo = min(max(first - before, 0), mine);
      const int hi = min(max(last - before, 0), mine);
      n[0] = min(n[0], hi);
      n[1] = min(n[1], hi);
    }
    if constexpr (kCut) ctl->t_lo[lane] = lo;
    ctl->n_tiles[0][lane] = n[0];
    ctl->n_tiles[1][lane] = n[1];
  }
  if (warp == 8) {
    tmem_alloc(&ctl->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (a.overlap) grid_dependency_wait();

  const uint32_t tmem = ctl->tmem_base;  // columns: S [0,128) P0 [128,192) P1 [192,256) O0 [256,384) O1 [384,512)

  bool any_work = false;
  for (int s = 0; s < a.nseg; ++s) any_work |= seg_tiles(ctl, s) > seg_first<kCut>(ctl, s);

  // Registers move from the auxiliary warpgroup (warps 8-11) to the two softmax
  // warpgroups; each role changes its own budget as the first thing it does.
  if (warp == 11) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 " MB_STR(MB_FWD_AUX_REGS) ";");
  } else if (warp == 9) {
    // ------------------------------------------------------------------ loader
    asm volatile("setmaxnreg.dec.sync.aligned.u32 " MB_STR(MB_FWD_AUX_REGS) ";");
    if (lane == 0 && any_work) {
      bool ok = true;
      const CUtensorMap* qmap = &maps.q[J.qmap];
      tma_prefetch_desc(qmap);
      if (J.q_flag != nullptr) {
        // The queries are being staged from another GPU: wait (bounded) for their arrival flag.  On a
        // timeout the Q load is skipped; every other role then runs into the abort word and returns.
        ok = flag_wait_ge(J.q_flag, J.q_flag_value, abort_word, MB_ERR_TIMEOUT_SEGMENT, a.peer_wait_cycles);
        asm volatile("fence.proxy.async;" ::: "memory");
      }
      if (ok) {
        const int rows = J.Sq << pack_shift;
        const int act0 = q0 < rows, act1 = q0 + kBM < rows;
        mbar_expect_tx(&ctl->q_full, (act0 + act1) * kTileBytes);
        for (int i = 0; i < 2; ++i) {
          if (q0 + i * kBM < rows) {
            const int r0 = (q0 + i * kBM) >> pack_shift;
            tma_load_4d(sQ + i * kTileBytes, qmap, &ctl->q_full, 0, ctl->h, r0, ctl->b);
            tma_load_4d(sQ + i * kTileBytes + kHalfBytes, qmap, &ctl->q_full, 64, ctl->h, r0, ctl->b);
          }
        }
      }
      int n = 0;
      const int b_ = ctl->b, hkv = ctl->h / a.group;
      // One K or V tile into the next stage of the ring.
      auto load_tile = [&](int which, const TileIter& it) {
        if (which == 0 && it.jt == seg_first<kCut>(ctl, it.s) && a.seg_flag[it.s] != nullptr) {
          // The shard is being staged by another stream: wait (bounded) for its arrival flag,
          // then order the TMA reads (async proxy) after the flag read.
          ok = flag_wait_ge(a.seg_flag[it.s], a.seg_flag_value[it.s], abort_word, MB_ERR_TIMEOUT_SEGMENT,
                            a.peer_wait_cycles);
          asm volatile("fence.proxy.async;" ::: "memory");
          if (!ok) return;
        }
        const int stage = n % kFwdStages;
        const int round = n / kFwdStages;
        if (round > 0 && !mbar_wait(&ctl->kv_empty[stage], (round - 1) & 1, abort_word, MB_ERR_TIMEOUT_KV_EMPTY, a.wait_cycles)) {
          ok = false;
          return;
        }
        const CUtensorMap* map = which ? &maps.v[it.s] : &maps.k[it.s];
        uint8_t* dst = sKV + stage * kTileBytes;
        mbar_expect_tx(&ctl->kv_full[stage], kTileBytes);
        tma_load_4d(dst, map, &ctl->kv_full[stage], 0, hkv, it.jt * kBN, b_);
        tma_load_4d(dst + kHalfBytes, map, &ctl->kv_full[stage], 64, hkv, it.jt * kBN, b_);
        ++n;
      };
      TileIter nxt = iter_first<kCut>(ctl, a.nseg);
      TileIter cur = nxt;
      if (ok && nxt.s < a.nseg) {
        load_tile(0, nxt);
        iter_next<kCut>(ctl, a.nseg, nxt);
      }
      while (ok && cur.s < a.nseg) {
        if (nxt.s < a.nseg) load_tile(0, nxt);
        if (ok) load_tile(1, cur);
        cur = nxt;
        if (nxt.s < a.nseg) iter_next<kCut>(ctl, a.nseg, nxt);
      }
      if (!ok) {
        // Give copies already in flight a bounded chance to land before the CTA exits.
        const int first = n > kFwdStages ? n - kFwdStages : 0;
        for (int m = first; m < n; ++m) {
          const long long t0 = clock64();
          while (!mbar_try_wait(&ctl->kv_full[m % kFwdStages], (m / kFwdStages) & 1) &&
                 clock64() - t0 < kWaitCycleLimit / 16) {
          }
        }
      }
    }
  } else if (warp == 8 || warp == 10) {
    // ------------------------------------------- MMA issuers: warp 8 issues every Q.K^T product,
    // warp 10 every P.V product, of both query tiles.  (One warp per query tile issuing both kinds
    // held its P.V products back while it sat in the issue of its next score product, and the
    // products of the two tiles then fell into the same stretch of time, with the tensor pipe idle
    // in between.)  Positions in the ring of K/V stages follow the load order K0 K1 V0 K2 V1 ...
    asm volatile("setmaxnreg.dec.sync.aligned.u32 " MB_STR(MB_FWD_AUX_REGS) ";");
    if (any_work) {  // whole warp, converged
      constexpr uint32_t kStageUnits = kTileBytes / 16;
      int total = 0;  // K/V tiles this CTA walks through
      for (int s = 0; s < a.nseg; ++s) total += max(seg_tiles(ctl, s) - seg_first<kCut>(ctl, s), 0);
      bool ok = true;
      if (warp == 8) {
        constexpr uint32_t idesc_qk = umma_idesc_bf16(kBM, kBN, false, false);
        const uint64_t q_desc = umma_smem_desc(smem_u32(sQ), 16, 1024);
        const uint64_t k_desc0 = umma_smem_desc(smem_u32(sKV), 16, 1024);  // K-major view of stage 0
        int g = 0;    // K/V tile index over all segments
        int use = 0;  // uses of the score region so far, by either query tile
        ok = mbar_wait_warp(&ctl->q_full, 0, abort_word, MB_ERR_TIMEOUT_Q, a.wait_cycles);
        for (int s = 0; s < a.nseg && ok; ++s) {
          const int n0 = ctl->n_tiles[0][s], n1 = ctl->n_tiles[1][s];
          const int nmax = max(n0, n1);
          for (int jt = seg_first<kCut>(ctl, s); jt < nmax && ok; ++jt, ++g) {
            const int pos = g == 0 ? 0 : 2 * g - 1;
            const int stage = pos % kFwdStages;
            ok = mbar_wait_warp(&ctl->kv_full[stage], (pos / kFwdStages) & 1, abort_word, MB_ERR_TIMEOUT_KV_FULL, a.wait_cycles);
            if (!ok) break;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if (jt < (i ? n1 : n0)) {
                // the score region's previous user must have copied its scores out
                if (use > 0) {
                  ok = mbar_wait_warp(&ctl->s_free, (use - 1) & 1, abort_word, MB_ERR_TIMEOUT_S, a.wait_cycles);
                  if (!ok) break;
                }
                tc_fence_after();
                issue_qk(tmem, q_desc + i * kStageUnits, k_desc0 + stage * kStageUnits, idesc_qk);
                umma_commit_elect(&ctl->s_full[i]);
                ++use;
              }
            }
            if (!ok) break;
            umma_commit_elect(&ctl->kv_empty[stage]);
          }
        }
      } else {
        constexpr uint32_t idesc_pv = umma_idesc_bf16(kBM, kD, false, true);
        const uint64_t v_desc0 = umma_smem_desc(smem_u32(sKV), kHalfBytes, 1024);  // MN-major view of stage 0
        int g = 0;
        int cnt0 = 0, cnt1 = 0;  // P.V products issued per query tile
        for (int s = 0; s < a.nseg && ok; ++s) {
          const int n0 = ctl->n_tiles[0][s], n1 = ctl->n_tiles[1][s];
          const int nmax = max(n0, n1);
          for (int jt = seg_first<kCut>(ctl, s); jt < nmax && ok; ++jt, ++g) {
            const int pos = g == total - 1 ? 2 * total - 1 : 2 * g + 2;
            const int stage = pos % kFwdStages;
            ok = mbar_wait_warp(&ctl->kv_full[stage], (pos / kFwdStages) & 1, abort_word, MB_ERR_TIMEOUT_KV_FULL, a.wait_cycles);
            if (!ok) break;
            const uint64_t v_desc = v_desc0 + stage * kStageUnits;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if (jt < (i ? n1 : n0)) {
                const int cnt = i ? cnt1 : cnt0;
                const uint32_t tPi = tmem + 128 + i * 64, tOi = tmem + 256 + i * 128;
                ok = mbar_wait_warp(&ctl->p_full[i][0], cnt & 1, abort_word, MB_ERR_TIMEOUT_P, a.wait_cycles);
                if (!ok) break;
                tc_fence_after();
                issue_pv_half(tOi, tPi, v_desc, idesc_pv, (cnt == 0 && !J.st_in) ? 0u : 1u);
                ok = mbar_wait_warp(&ctl->p_full[i][1], cnt & 1, abort_word, MB_ERR_TIMEOUT_P, a.wait_cycles);
                if (!ok) break;
                tc_fence_after();
                issue_pv_half(tOi, tPi + 32, v_desc + 4 * 128, idesc_pv, 1u);
                umma_commit_elect(&ctl->o_full[i]);
                if (i) ++cnt1;
                else ++cnt0;
              }
            }
            if (!ok) break;
            umma_commit_elect(&ctl->kv_empty[stage]);
          }
        }
      }
      if (!ok) {
        // Let tensor-core work already issued finish (bounded) before tensor memory is released.
        umma_commit_elect(&ctl->drain);
        const long long t0 = clock64();
        while (!mbar_try_wait(&ctl->drain, 0) && clock64() - t0 < kWaitCycleLimit / 16) {
        }
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------ softmax + epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 " MB_STR(MB_FWD_SOFTMAX_REGS) ";");
    // All control flow below is warp-uniform (the tensor-memory loads and
    // stores are warp-collective); only global stores are predicated per row.
    const int i = warp >> 2;                    // query tile
    const int row = ((warp & 3) << 5) | lane;   // row inside the tile == tensor-memory lane
    const uint32_t lane_field = static_cast<uint32_t>((warp & 3) << 5) << 16;
    const uint32_t tS = tmem + lane_field;
    const uint32_t tPi = tmem + 128 + i * 64 + lane_field;
    const uint32_t tOi = tmem + 256 + i * 128 + lane_field;
    // global position used by the causal rule (of the tile's first row: qfirst); the row inside the job's Q is
    // qpos - J.q_off
    const int qfirst = J.q_off + ((q0 + i * kBM) >> pack_shift);
    const int qpos = qfirst + (row >> pack_shift);

    float m_ref = -INFINITY;  // reference max (raw score units)
    float l = 0.f;            // running sum of exp2
    int cnt = 0;
    bool ok = true;
    if (J.st_in && q0 + i * kBM < J.Sq) {  // (carried states go with unpacked rows)
      const int qrow = qpos - J.q_off;  // row inside the job's Q
      const long long st_row = ((long long)ctl->b * a.Hq + ctl->h) * J.Sq + qrow;
      // Continue where an earlier job stopped: its unnormalised rows go back into tensor memory, its
      // maximum and sum into registers.  With chain words that job may be part of this launch (a CTA
      // with a lower index); its release store is acquired here.
      if (J.chain != nullptr) {
        if (lane == 0)
          ok = flag_wait_ge(J.chain + ((long long)ctl->b * a.Hq + ctl->h) * J.n_pairs + ctl->pair, J.chain_wait, abort_word,
                            MB_ERR_TIMEOUT_SEGMENT, a.peer_wait_cycles);
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      }
      if (ok) {
        const bool valid = qrow < J.Sq;
        const float4* src = reinterpret_cast<const float4*>(J.st_o + st_row * kD);
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t orow[32];
#pragma unroll
          for (int v = 0; v < 8; ++v) {
            const float4 w = valid ? src[c * 8 + v] : make_float4(0.f, 0.f, 0.f, 0.f);
            orow[v * 4 + 0] = __float_as_uint(w.x);
            orow[v * 4 + 1] = __float_as_uint(w.y);
            orow[v * 4 + 2] = __float_as_uint(w.z);
            orow[v * 4 + 3] = __float_as_uint(w.w);
          }
          tmem_st32(tOi + c * 32, orow);
        }
        tmem_wait_st();
        if (valid) {
          const float2 ml = *reinterpret_cast<const float2*>(J.st_ml + st_row * 2);
          m_ref = ml.x;
          l = ml.y;
        }
      }
    }

    for (int s = 0; s < a.nseg && ok; ++s) {
      const int nt = ctl->n_tiles[i][s];
      const int sk = a.seg_sk[s];
      const int koff = a.seg_koff[s];
      for (int jt = seg_first<kCut>(ctl, s); jt < nt; ++jt) {
        ok = mbar_wait_warp(&ctl->s_full[i], cnt & 1, abort_word, MB_ERR_TIMEOUT_S, a.wait_cycles);
        if (!ok) break;
        tc_fence_after();
        uint32_t sr[4][32];
        tmem_ld32(tS + 0, sr[0]);
        tmem_ld32(tS + 32, sr[1]);
        tmem_ld32(tS + 64, sr[2]);
        tmem_ld32(tS + 96, sr[3]);
        tmem_wait_ld();
        // The scores are in registers: hand the score region to its next user.
        tc_fence_before();
        mbar_arrive_elect(&ctl->s_free);

        // masking: only tiles that cross the segment end or the causal diagonal
        const int k0 = jt * kBN;
        const bool tile_needs_mask =
            (k0 + kBN > sk) || (a.causal && (koff + k0 + kBN - 1 > qfirst));
        if (tile_needs_mask) {
          int limit = sk - k0;  // columns >= limit are invisible
          if (a.causal) limit = min(limit, qpos - koff - k0 + 1);
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (c * 32 + e >= limit) sr[c][e] = 0xff800000u;  // -inf
        }

        float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          mx0 = max3(mx0, __uint_as_float(sr[0][e]), __uint_as_float(sr[0][e + 1]));
          mx1 = max3(mx1, __uint_as_float(sr[1][e]), __uint_as_float(sr[1][e + 1]));
          mx2 = max3(mx2, __uint_as_float(sr[2][e]), __uint_as_float(sr[2][e + 1]));
          mx3 = max3(mx3, __uint_as_float(sr[3][e]), __uint_as_float(sr[3][e + 1]));
        }
        const float m_tile = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));

        if (cnt == 0 && __all_sync(0xffffffffu, m_ref == -INFINITY)) {
          m_ref = m_tile;  // nothing accumulated yet (a carried state of rows without keys is all zero)
        } else {
          // The previous P.V product of this query tile must be complete before its probabilities
          // are overwritten, and before O is rescaled (a carried state is already in place).
          if (cnt > 0) {
            ok = mbar_wait_warp(&ctl->o_full[i], (cnt - 1) & 1, abort_word, MB_ERR_TIMEOUT_O, a.wait_cycles);
            if (!ok) break;
            tc_fence_after();
          }
          const float m_new = fmaxf(m_ref, m_tile);
          const bool need = (m_new - m_ref) * a.scale_log2 > kRescaleThreshold;
          if (__any_sync(0xffffffffu, need)) {
            const float f = need ? fast_exp2((m_ref - m_new) * a.scale_log2) : 1.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              uint32_t orow[32];
              tmem_ld32(tOi + c * 32, orow);
              tmem_wait_ld();
#pragma unroll
              for (int e = 0; e < 32; ++e) orow[e] = __float_as_uint(__uint_as_float(orow[e]) * f);
              tmem_st32(tOi + c * 32, orow);
            }
            tmem_wait_st();
            if (need) {
              l *= f;
              m_ref = m_new;
            }
          }
        }

        // p = exp2(s * c - m * c): the scale/subtract and the row sum run as packed pairs.  (Taking
        // turns between the two warpgroups in this MUFU-bound phase, and moving part of the
        // exponentials to a polynomial on the FMA pipe, were both measured as losses.)
        const float m_scaled = (m_ref == -INFINITY) ? 0.f : m_ref * a.scale_log2;
        const uint64_t c2 = pack2(a.scale_log2, a.scale_log2);
        const uint64_t nm2 = pack2(-m_scaled, -m_scaled);
        uint64_t sum_a = pack2(0.f, 0.f), sum_b = pack2(0.f, 0.f);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t pk[32];
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            const int c = half * 2 + cc;
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
              const uint64_t x2 = fma2(pack2(__uint_as_float(sr[c][e]), __uint_as_float(sr[c][e + 1])), c2, nm2);
              float x0, x1;
              unpack2(x2, x0, x1);
              const uint64_t p2 = pack2(fast_exp2(x0), fast_exp2(x1));
              if ((e >> 1) & 1) sum_b = add2(sum_b, p2);
              else sum_a = add2(sum_a, p2);
              float p0, p1;
              unpack2(p2, p0, p1);
              pk[cc * 16 + (e >> 1)] = pack_bf16x2(p0, p1);
            }
          }
          tmem_st32(tPi + half * 32, pk);
          tmem_wait_st();
          tc_fence_before();
          mbar_arrive(&ctl->p_full[i][half]);
        }
        {
          float s0, s1;
          unpack2(add2(sum_a, sum_b), s0, s1);
          l += s0 + s1;
        }
        ++cnt;
      }
    }

    // epilogue.  Final job: O / l -> bf16, LSE = ln(sum exp(scale * s)).  Job that hands its state on:
    // the unnormalised rows, the maximum and the sum, as they are.  Tiles whose rows all lie past Sq skip it.
    const int qrow = qpos - J.q_off;  // row inside the job's Q
    if (ok && qfirst - J.q_off < J.Sq) {
      const long long st_row = ((long long)ctl->b * a.Hq + ctl->h) * J.Sq + qrow;
      const bool have_acc = cnt > 0 || J.st_in;   // tensor memory holds this tile's rows
      if (cnt > 0) ok = mbar_wait_warp(&ctl->o_full[i], (cnt - 1) & 1, abort_word, MB_ERR_TIMEOUT_O, a.wait_cycles);
      if (ok) {
        const bool store = qrow < J.Sq;
        if (have_acc) tc_fence_after();
        if (kCut && ctl->slot >= 0) {
          // a share of the item: rows as they are, column group by column group (contiguous over a warp)
          const int r = i * kBM + row;
          if (cnt > 0) {
            float4* dst = a.part_o + (long long)ctl->slot * (32 * 2 * kBM) + r;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              uint32_t orow[32];
              tmem_ld32(tOi + c * 32, orow);
              tmem_wait_ld();
#pragma unroll
              for (int v = 0; v < 8; ++v)
                dst[(c * 8 + v) * (2 * kBM)] =
                    make_float4(__uint_as_float(orow[v * 4 + 0]), __uint_as_float(orow[v * 4 + 1]),
                                __uint_as_float(orow[v * 4 + 2]), __uint_as_float(orow[v * 4 + 3]));
            }
          }
          a.part_ml[ctl->slot * (2 * kBM) + r] = make_float2(m_ref, l);
        } else if (J.st_out) {
          float4* dst = reinterpret_cast<float4*>(J.st_o + st_row * kD);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t orow[32];
            if (have_acc) {
              tmem_ld32(tOi + c * 32, orow);
              tmem_wait_ld();
            } else {
#pragma unroll
              for (int e = 0; e < 32; ++e) orow[e] = 0u;
            }
            if (store) {
#pragma unroll
              for (int v = 0; v < 8; ++v)
                dst[c * 8 + v] = make_float4(__uint_as_float(orow[v * 4 + 0]), __uint_as_float(orow[v * 4 + 1]),
                                             __uint_as_float(orow[v * 4 + 2]), __uint_as_float(orow[v * 4 + 3]));
            }
          }
          if (store) *reinterpret_cast<float2*>(J.st_ml + st_row * 2) = make_float2(m_ref, l);
        } else {
          const float inv_l = (have_acc && l > 0.f) ? 1.f / l : 0.f;
          const int head = ctl->h + (row & ((1 << pack_shift) - 1));
          __nv_bfloat16* optr = J.o + (long long)ctl->b * J.o_sb + (long long)qrow * J.o_ss + (long long)head * J.o_sh;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t orow[32];
            if (have_acc) {
              tmem_ld32(tOi + c * 32, orow);
              tmem_wait_ld();
            } else {
#pragma unroll
              for (int e = 0; e < 32; ++e) orow[e] = 0u;
            }
            if (store) {
              uint4* dst = reinterpret_cast<uint4*>(optr + c * 32);
#pragma unroll
              for (int v = 0; v < 4; ++v) {
                uint4 w;
                w.x = pack_bf16x2(__uint_as_float(orow[v * 8 + 0]) * inv_l, __uint_as_float(orow[v * 8 + 1]) * inv_l);
                w.y = pack_bf16x2(__uint_as_float(orow[v * 8 + 2]) * inv_l, __uint_as_float(orow[v * 8 + 3]) * inv_l);
                w.z = pack_bf16x2(__uint_as_float(orow[v * 8 + 4]) * inv_l, __uint_as_float(orow[v * 8 + 5]) * inv_l);
                w.w = pack_bf16x2(__uint_as_float(orow[v * 8 + 6]) * inv_l, __uint_as_float(orow[v * 8 + 7]) * inv_l);
                dst[v] = w;
              }
            }
          }
          if (store) {
            const float lse = (have_acc && l > 0.f) ? (m_ref * a.scale + __logf(l)) : -INFINITY;
            J.lse[(long long)ctl->b * J.lse_sb + (long long)head * J.lse_sh + qrow] = lse;
          }
        }
      }
    }
    if (J.st_out && J.chain != nullptr) {
      // Publish the state to the job that continues it: every softmax thread's stores, then one release
      // store of the chain word.  (A CTA that gave up publishes too, so that nothing downstream waits out
      // its budget; the status word tells the host.)
      __threadfence();
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (warp == 0 && lane == 0)
        asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(J.chain + ((long long)ctl->b * a.Hq + ctl->h) * J.n_pairs + ctl->pair),
                     "r"(J.chain_set)
                     : "memory");
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  if (tid == 0 && ctl->abort_word != 0 && a.status != nullptr) atomicCAS(a.status, 0, ctl->abort_word);
  if (tid == 0 && J.done_flag != nullptr) {
    // Every thread's result stores precede the barrier above; this fence makes them visible at system
    // scope (they may have gone to another GPU) before the arrival is counted.  The CTA that counts the
    // last arrival publishes the job: the flag's reader then sees every row of every CTA.  A CTA that
    // gave up still counts, so that the word returns to zero; the status word tells the host.
    __threadfence_system();
    int prev;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(prev) : "l"(J.done_counter) : "memory");
    if (prev == J.n_ctas - 1) {
      *J.done_counter = 0;
      __threadfence_system();
      asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(J.done_flag), "r"(J.done_value) : "memory");
    }
  }
}

// ---------------------------------------------------------------------------
// split items: the shares of an item become its result
// ---------------------------------------------------------------------------
struct FwdMergeArgs {
  const float4* part_o;  // [slot][32 column groups][256 rows]
  const float2* part_ml;
  __nv_bfloat16* o;
  long long o_sb, o_ss, o_sh;
  float* lse;
  long long lse_sb, lse_sh;
  int Sq, B, Hq, n_pairs, pack_shift, head_block, causal, first_item, nsplit;
  float scale, scale_log2;
};

// o = sum_p w_p O_p / sum_p w_p l_p with w_p = exp(scale * (m_p - max m)), in fp32.  A block handles 8 rows: warp w
// columns [16 w, 16 w + 16), a lane 4 columns of one row, so that the lanes of a column group read 128 contiguous
// bytes of a share and a row's 16 bf16 results are one 32-byte sector.  Latency-bound (the shares are in L2), hence
// many small blocks and few registers.  After an attention launch of one wave its blocks are set up under the end of that
// kernel; a longer one does not trigger it early (see launch_fwd) and is drained first.
constexpr int kMergeRows = 8;
__global__ void __launch_bounds__(256) fwd_split_merge_kernel(const FwdMergeArgs a) {
  constexpr int kRows = 2 * kBM;
  const int lane = threadIdx.x & 31, chunk = (threadIdx.x >> 5) * 4 + (lane >> 3);  // group of 4 columns
  const int item = blockIdx.x;
  const int r = blockIdx.y * kMergeRows + (lane & 7);
  const ItemCoords it = item_coords(a.first_item + item, a.n_pairs, a.head_block, a.B, a.Hq >> a.pack_shift, a.causal);
  const int prow = it.pair * kRows + r;  // row over (query, head of the group)
  const int qrow = prow >> a.pack_shift, head = (it.h << a.pack_shift) + (prow & ((1 << a.pack_shift) - 1));
  grid_dependents_launch();
  grid_dependency_wait();
  if (qrow >= a.Sq) return;
  const long long slot0 = (long long)item * a.nsplit;
  const float2* ml = a.part_ml + slot0 * kRows + r;
  float m = -INFINITY;
#pragma unroll 8
  for (int p = 0; p < a.nsplit; ++p) m = fmaxf(m, ml[p * kRows].x);
  float l = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
  const float4* src = a.part_o + (slot0 * 32 + chunk) * kRows + r;
#pragma unroll 8
  for (int p = 0; p < a.nsplit; ++p) {
    const float2 s = ml[p * kRows];
    const bool has = !(s.y == 0.f);  // a share without visible keys has stored no rows
    const float4 x = has ? src[(long long)p * 32 * kRows] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float w = has ? fast_exp2((s.x - m) * a.scale_log2) : 0.f;
    l = fmaf(w, s.y, l);
    acc[0] = fmaf(w, x.x, acc[0]);
    acc[1] = fmaf(w, x.y, acc[1]);
    acc[2] = fmaf(w, x.z, acc[2]);
    acc[3] = fmaf(w, x.w, acc[3]);
  }
  const float inv = l > 0.f ? 1.f / l : 0.f;
  uint2 o;
  o.x = pack_bf16x2(acc[0] * inv, acc[1] * inv);
  o.y = pack_bf16x2(acc[2] * inv, acc[3] * inv);
  *reinterpret_cast<uint2*>(a.o + it.b * a.o_sb + qrow * a.o_ss + head * a.o_sh + chunk * 4) = o;
  if (chunk == 0) a.lse[it.b * a.lse_sb + head * a.lse_sh + qrow] = l > 0.f ? m * a.scale + __logf(l) : -INFINITY;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// How a single-job launch is cut: items before split_begin run whole, the others as nsplit shares each.
struct FwdSplit {
  int split_begin, nsplit, slots;
};
constexpr FwdSplit kWhole{INT_MAX, 1, 0};
constexpr size_t kSlotBytes = 2 * kBM * (kD * sizeof(float) + sizeof(float2));

int sm_count() {
  static int count[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (count[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    count[dev] = n;
  }
  return count[dev];
}

// log2 of the query heads that share a tile row by row (row = query * heads + head).  The heads of a group read the
// same K/V, so a tile of 128 rows may hold all of them for 128 / group queries instead of one of them for 128:
// worth it when the queries of one head leave much of a pair of tiles empty, which is where it saves an eighth of the
// pairs.  Grouped layouts only, groups that divide a tile.  Measured (B200): 100 queries against 16 384 keys, 32
// heads over 8: 55 us head by head (32 pairs, half empty), 42 us packed (16 pairs).
static int plan_pack(int sq, int hq, int hkv) {
  if (hkv <= 0 || hq % hkv != 0) return 0;
  const int group = hq / hkv;
  int shift = 0;
  while ((1 << shift) < group && shift < 8) ++shift;
  if ((1 << shift) != group || group > kBM || sq > INT_MAX / group - 2 * kBM) return 0;
  const long long apart = (long long)group * ((sq + 2ll * kBM - 1) / (2 * kBM));  // pairs of a group, head by head
  const long long packed = ((long long)sq * group + 2 * kBM - 1) / (2 * kBM);
  return packed * 8 <= apart * 7 ? shift : 0;
}

// K/V tiles that a pair of query tiles walks through.
static long long pair_tiles(const mb_attn_fwd_args* x, int pack_shift, int pair) {
  const long long row = min(((pair + 1ll) * 2 * kBM - 1) >> pack_shift, x->sq - 1ll);  // the pair's last one
  long long t = 0;
  for (int s = 0; s < x->nseg; ++s) {
    long long vis = x->seg[s].sk;
    if (x->causal) vis = min(vis, x->q_off + row - x->seg[s].k_off + 1);
    if (vis > 0) t += (vis + kBN - 1) / kBN;
  }
  return t;
}

// Without a split a launch of few items runs on as many SMs as it has items, and a last wave of few items leaves the
// others idle.  Measured (B200), whole / split: 128 queries against 2 048 keys, 8 heads, 27 / 17 us; against 32 768 keys,
// 315 / 41 us; 1 024 causal rows, 8 heads, 21 / 19 us; 4 096 queries against 32 768 keys, 32 heads (3.46 waves),
// 1.92 / 1.80 ms with the last 68 items in 2 shares; 5 000 x 5 000, 16 heads, 234 / 188 us.  Shapes that the
// costs below leave whole, and what a split did to them: 768 x 768, 8 heads, in 6 shares 19 -> 21 us; 2 048 x 4 096, 32
// heads (108 items in the last wave), in 4 shares 132 -> 145 us.
static FwdSplit plan_split(const mb_attn_fwd_args* x, int pack_shift) {
  const FwdSplit whole = kWhole;
  if (x->sq <= 0 || x->softmax_scale <= 0.f) return whole;
  const int sms = sm_count();
  const int np = ((x->sq << pack_shift) + 2 * kBM - 1) / (2 * kBM), heads = x->hq >> pack_shift;
  const long long items = (long long)np * heads * x->batch;
  if (sms <= 0 || items > INT_MAX) return whole;
  // Several shards: only the last wave of a non-causal launch is split.  Smaller launches and causal ones stay whole for
  // callers that compare them with chained jobs (mb_attn_fwd_multi) bit for bit; what that costs, measured
  // against one segment with the same keys: 256 queries, 8 heads, 8 shards of 256 keys 51 / 24 us, of 4 096
  // keys 381 / 46 us; 1 024 causal rows, 8 shards of 1 024 keys 68 / 29 us.  From one wave up the equality
  // holds for the whole items only.
  if (x->nseg > 1 && (x->causal || items < sms)) return whole;
  for (int s = 0; s < x->nseg; ++s)
    if (x->seg[s].ready_flag != nullptr) return whole;
  // K/V tiles of the longest item, of the shortest one and of all items of a head
  long long t_max = 0, t_min = 0, t_sum = 0;
  if (!x->causal) t_max = pair_tiles(x, pack_shift, 0);
  if (x->causal) {
    if (items > 4ll * sms) return whole;
    t_min = LLONG_MAX;
    for (int p = 0; p < np; ++p) {
      const long long t = pair_tiles(x, pack_shift, p);
      t_max = max(t_max, t);
      t_min = min(t_min, t);
      t_sum += t;
    }
  }
  // Costs in steps of one K/V tile against both query tiles (1.7 us): starting and ending a CTA, the extra launch
  // that merges the shares, and per share its way through memory.  A wave that leaves SMs idle is also faster
  // per step (the chip clocks higher): 0.8 of a full one where 68 of 148 SMs work.
  constexpr double kCta = 1.25, kMerge = 2.0, kSlot = 0.02;
  constexpr int kMaxSplit = 32;
  auto pace = [&](double busy) { return 0.65 + 0.35 * busy / sms; };
  const long long slot_cap = 3ll * sms;
  FwdSplit best = whole;
  if (x->causal) {
    // Items of unequal length, longest first: one after the other on every SM until the shortest ones fill up
    // the end, unless there are fewer items than SMs.
    const double total = (double)t_sum * heads * x->batch;
    auto cost = [&](int ns) {
      const double longest = (double)((t_max + ns - 1) / ns) + kCta;
      if (items * ns <= sms) return longest;
      return max(longest, (total + items * ns * kCta) / sms + (double)t_min / ns + kCta);
    };
    // Shares of more than one wave cost more than that: the merge waits for the launch to drain, and the shares of
    // the third wave start late.  Measured less the sum above: 4 to 5 steps with 192 to 288 shares, 5 to 10 with
    // 304 to 384.  8 heads, causal, whole / 2 shares: 4 352 rows 60.1 / 56.8 us, 4 864 (304 shares) 66.7 / 70.0,
    // 5 000 68.8 / 74.3, 6 144 82.7 / 98.3; 4 heads, 9 728 rows 122.5 / 99.2.
    auto late = [&](long long shares) { return shares > 2 * sms ? 7.5 : shares > sms ? 4.5 : 0.0; };
    double t_best = cost(1);
    for (int ns = 2; ns <= kMaxSplit && ns <= t_max && items * ns <= slot_cap; ++ns) {
      const double t = cost(ns) + kMerge + kSlot * items * ns + late(items * ns);
      if (t < t_best) {
        t_best = t;
        best = FwdSplit{0, ns, (int)(items * ns)};
      }
    }
  } else {
    // Equal items: whole waves run as they are, the items of the last, partly filled one are split.
    const int rest = (int)(items % sms);
    double t_best = t_max * pace(rest) + kCta;
    for (int ns = 2; rest > 0 && ns <= kMaxSplit && ns <= t_max && (long long)rest * ns <= slot_cap; ++ns) {
      const int waves = (rest * ns + sms - 1) / sms;
      const double t = waves * ((t_max + ns - 1) / ns * pace((double)rest * ns / waves) + kCta) + kMerge + kSlot * rest * ns;
      if (t < t_best) {
        t_best = t;
        best = FwdSplit{(int)(items - rest), ns, rest * ns};
      }
    }
  }
  return best;
}

struct FwdPlan {
  int pack_shift;
  FwdSplit split;
};

// Heads are packed where plan_pack says so and the launch is split, or has more than one wave of pairs when the heads
// stay apart.  Whole launches of one wave last as long as their longest pair, and a packed pair is a full one: only
// where that pair has both tiles anyway and many steps does the smaller number of busy SMs (which clock higher)
// make up for it.  Measured (B200), packed / apart: 4 x 128 x 128, 32 heads over 8, 9.2 / 7.4 us; 2 x 889 x 889
// causal, 16 over 4, 18.9 / 17.1; 586 causal rows in 4 shards, 8 over 2, 31.0 / 29.3; 2 x 392 x 20 030 causal, 32
// over 8, 248 / 255.  Non-causal launches of more waves need a fifth of the pairs saved (32 heads over 8: 4 x 440 x
// 440, 256 -> 224 pairs, 30.3 / 28.9; 4 x 300 x 300, 256 -> 160, 24.7 / 26.7), causal ones, whose pairs are of many
// lengths, do not (8 x 440 x 440, 512 -> 448, 43.2 / 46.7).
static FwdPlan plan_fwd(const mb_attn_fwd_args* x, bool may_split) {
  FwdPlan p{plan_pack(x->sq, x->hq, x->hkv), kWhole};
  if (x->sq <= 0) return FwdPlan{0, kWhole};
  if (may_split) p.split = plan_split(x, p.pack_shift);
  if (p.pack_shift == 0 || p.split.slots > 0) return p;
  const long long np = (x->sq + 2ll * kBM - 1) / (2 * kBM);
  bool apart = false;
  if (np * x->hq * x->batch <= sm_count()) {
    const int rows = x->causal ? (x->sq - 1) % (2 * kBM) + 1 : min(x->sq, 2 * kBM);  // of the longest pair
    apart = rows <= kBM || pair_tiles(x, 0, (int)np - 1) < 16;
  } else if (!x->causal) {
    const long long packed = (((long long)x->sq << p.pack_shift) + 2 * kBM - 1) / (2 * kBM);
    apart = packed * 5 > (np << p.pack_shift) * 4;
  }
  if (apart) p = FwdPlan{0, may_split ? plan_split(x, 0) : kWhole};
  return p;
}

long long attn_fwd_workspace(const mb_attn_fwd_args* x) {
  if (x == nullptr || x->nseg < 0 || x->nseg > MB_MAX_SEGMENTS || x->hq <= 0 || x->batch <= 0) return 0;
  return plan_fwd(x, true).split.slots * (long long)kSlotBytes;
}

constexpr long long kL2Bytes = 64ll << 20;
// Heads whose items are dispatched together, longest first, in a causal launch: as many as have their K/V in kL2Bytes
// of L2, in equal blocks.  Head by head, the longest items of the last heads start when most of the work is
// done and the launch waits for them.  Measured (B200): batch 2, 2 999 rows, 16 heads over 4: 107 us head by
// head, 92 us over all heads; 32 768 rows, 32 heads (16 MiB a head): 16, 32, 64 and 128 MiB alike within 1 %.
static int causal_head_block(const FwdArgs& a) {
  long long rows = 0;
  for (int s = 0; s < a.nseg; ++s) rows += a.seg_sk[s];
  const long long kv_bytes = max(rows * kD * 4, 1ll);  // K and V of one K/V head
  const long long heads = (long long)a.B * (a.Hq >> a.pack_shift);
  const long long fit = max(kL2Bytes / kv_bytes, 1ll) * (a.group >> a.pack_shift);
  if (fit >= heads) return (int)heads;
  const long long blocks = (heads + fit - 1) / fit;
  return (int)((heads + blocks - 1) / blocks);
}

static int make_tile_map(CUtensorMap* map, const void* ptr, int D, int H, int S, int B, long long sb, long long ss,
                         long long sh, int pack_shift = 0) {
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)sh * 2, (cuuint64_t)ss * 2, (cuuint64_t)sb * 2};
  cuuint32_t box[4] = {64, 1u << pack_shift, (cuuint32_t)kBN >> pack_shift, 1};  // 128 rows, heads innermost
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return encode_tiled_bf16(map, const_cast<void*>(ptr), 4, dims, strides, box, estr);
}

static long long g_peer_wait_ms = 30000;

void set_peer_wait_ms(unsigned ms) { g_peer_wait_ms = ms == 0 ? 1 : ms; }

// Cycle budget of waits for data other GPUs deliver: the SM clock never exceeds 2 GHz here, so
// 2e6 cycles per millisecond is at least the requested time.
long long peer_wait_cycles() { return g_peer_wait_ms * 2000000LL; }

// What a launch of one wave loses per K/V step of its CTAs (in steps) when it follows another under overlap, at `busy` of
// the SMs.  The two SMs of a TPC are slower when both work (64 steps: 103 us with up to 80 CTAs, 131 with 148).  An
// ordinary launch of few CTAs puts one on each TPC; under overlap they go where the launch before leaves SMs free,
// which comes out in pairs once the two together have more CTAs than SMs.  Measured back to back, overlapped / not,
// 128 steps: 48 CTAs 0.99, 64 1.01, 80 1.07, 92 1.06, 108 1.04, 124 1.01, 140 0.99; 20 steps: 72 CTAs 0.94, 80 1.02.
static double overlap_loss(double busy) {
  if (busy < 0.33 || busy > 0.95) return 0.0;
  return busy <= 0.5 ? 0.02 : 0.2 * (0.95 - busy);
}

// pack_shift != 0: one job without carried state or chain (see plan_pack).
static int launch_fwd(const mb_attn_fwd_multi_args* x, int pack_shift, const FwdSplit& split, void* ws,
                      cudaStream_t stream) {
  if (x == nullptr) return MB_E_INVALID;
  if (x->head_dim != kD) return MB_E_UNSUPPORTED;
  if (x->batch <= 0 || x->hq <= 0 || x->hkv <= 0 || x->hq % x->hkv != 0) return MB_E_INVALID;
  if (x->nseg < 0 || x->nseg > MB_MAX_SEGMENTS) return MB_E_INVALID;
  if (x->njobs < 1 || x->njobs > MB_MAX_JOBS) return MB_E_INVALID;

  static bool attr_set[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return MB_E_CUDA;
  if (dev < 64 && !attr_set[dev]) {
    if (cudaFuncSetAttribute(attn_fwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmemBytes) !=
            cudaSuccess ||
        cudaFuncSetAttribute(attn_fwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmemBytes) !=
            cudaSuccess)
      return MB_E_CUDA;
    attr_set[dev] = true;
  }

  // Kernel parameters (10.2 KB of tensor maps + 7.5 KB of jobs and scalars) are assembled in static storage:
  // the launch copies them, and launches of one process are issued from one thread at a time per device.
  static thread_local FwdMaps maps;
  static thread_local FwdArgs a;
  memset(&a, 0, sizeof(a));
  // empty segments are dropped; a job's segment mask is re-indexed accordingly
  int seg_new[MB_MAX_SEGMENTS];
  int nseg = 0;
  for (int s = 0; s < x->nseg; ++s) {
    const mb_kv_segment& g = x->seg[s];
    seg_new[s] = -1;
    if (g.sk < 0) return MB_E_INVALID;
    if (g.sk == 0) continue;  // an empty shard contributes nothing
    if (g.k == nullptr || g.v == nullptr) return MB_E_INVALID;
    if (make_tile_map(&maps.k[nseg], g.k, kD, x->hkv, g.sk, x->batch, g.stride_b, g.stride_s, g.stride_h))
      return MB_E_TENSORMAP;
    if (make_tile_map(&maps.v[nseg], g.v, kD, x->hkv, g.sk, x->batch, g.stride_b, g.stride_s, g.stride_h))
      return MB_E_TENSORMAP;
    a.seg_sk[nseg] = g.sk;
    a.seg_koff[nseg] = g.k_off;
    a.seg_flag[nseg] = g.ready_flag;
    a.seg_flag_value[nseg] = g.ready_value;
    seg_new[s] = nseg++;
  }
  a.nseg = nseg;
  int njobs = 0, x_total = 0, nqmaps = 0;
  const mb_fwd_job* qmap_of[kMaxQMaps];
  for (int j = 0; j < x->njobs; ++j) {
    const mb_fwd_job& g = x->job[j];
    if (g.sq < 0) return MB_E_INVALID;
    if (g.sq == 0) {
      // nothing to compute, but a completion flag must still be raised: only allowed without one
      if (g.done_flag != nullptr) return MB_E_INVALID;
      continue;
    }
    if (g.q == nullptr) return MB_E_INVALID;
    if (!g.state_out && (g.o == nullptr || g.lse == nullptr)) return MB_E_INVALID;
    if ((g.state_in || g.state_out) && (g.state_o == nullptr || g.state_ml == nullptr)) return MB_E_INVALID;
    if ((reinterpret_cast<uintptr_t>(g.state_o) & 15u) || (reinterpret_cast<uintptr_t>(g.state_ml) & 7u)) return MB_E_INVALID;
    if (g.done_flag != nullptr && g.done_counter == nullptr) return MB_E_INVALID;
    // jobs over the same query rows (the links of a state chain) share one tensor map
    int qmap = -1;
    for (int m = 0; m < nqmaps && qmap < 0; ++m) {
      const mb_fwd_job& o = *qmap_of[m];
      if (o.q == g.q && o.sq == g.sq && o.q_stride_b == g.q_stride_b && o.q_stride_s == g.q_stride_s &&
          o.q_stride_h == g.q_stride_h)
        qmap = m;
    }
    if (qmap < 0) {
      if (nqmaps == kMaxQMaps) return MB_E_INVALID;
      if (make_tile_map(&maps.q[nqmaps], g.q, kD, x->hq, g.sq, x->batch, g.q_stride_b, g.q_stride_s, g.q_stride_h,
                        pack_shift))
        return MB_E_TENSORMAP;
      qmap_of[nqmaps] = &g;
      qmap = nqmaps++;
    }
    FwdJob& J = a.job[njobs];
    J.qmap = qmap;
    J.o = reinterpret_cast<__nv_bfloat16*>(g.o);
    J.o_sb = g.o_stride_b;
    J.o_ss = g.o_stride_s;
    J.o_sh = g.o_stride_h;
    J.lse = g.lse;
    J.lse_sh = g.lse_stride_h ? g.lse_stride_h : g.sq;
    J.lse_sb = g.lse_stride_b ? g.lse_stride_b : (long long)x->hq * g.sq;
    J.Sq = g.sq;
    J.q_off = g.q_off;
    unsigned mask = 0;
    for (int s = 0; s < x->nseg; ++s)
      if (seg_new[s] >= 0 && (g.seg_mask == 0 || ((g.seg_mask >> s) & 1u))) mask |= 1u << seg_new[s];
    J.seg_mask = mask;
    J.x_begin = x_total;
    J.n_pairs = ((g.sq << pack_shift) + 2 * kBM - 1) / (2 * kBM);
    J.q_flag = g.q_ready_flag;
    J.q_flag_value = g.q_ready_value;
    J.done_flag = g.done_flag;
    J.done_value = g.done_value;
    J.done_counter = g.done_counter;
    J.n_ctas = J.n_pairs * (x->hq >> pack_shift) * x->batch;
    J.st_o = g.state_o;
    J.st_ml = g.state_ml;
    J.st_in = g.state_in ? 1 : 0;
    J.st_out = g.state_out ? 1 : 0;
    J.chain = g.chain;
    J.chain_wait = g.chain_wait;
    J.chain_set = g.chain_set;
    if (x_total > INT_MAX - J.n_ctas) return MB_E_INVALID;
    x_total += J.n_ctas;
    ++njobs;
  }
  if (njobs == 0) return MB_SUCCESS;
  a.njobs = njobs;
  a.B = x->batch;
  a.Hq = x->hq;
  a.group = x->hq / x->hkv;
  a.causal = x->causal ? 1 : 0;
  a.scale = x->softmax_scale;
  a.scale_log2 = x->softmax_scale * 1.4426950408889634f;
  a.peer_wait_cycles = peer_wait_cycles();
  bool has_flags = false;
  for (int s = 0; s < nseg; ++s) has_flags |= a.seg_flag[s] != nullptr;
  for (int j = 0; j < njobs; ++j) has_flags |= a.job[j].q_flag != nullptr || (a.job[j].chain != nullptr && a.job[j].st_in);
  a.wait_cycles = kWaitCycleLimit + (has_flags ? a.peer_wait_cycles : 0);
  a.status = x->status ? x->status : default_status_word();
  if (a.status == nullptr) return MB_E_CUDA;

  a.pack_shift = pack_shift;
  a.head_block = 1;
  if (a.causal && !has_flags && njobs == 1) a.head_block = causal_head_block(a);
  a.split_begin = split.split_begin;
  a.nsplit = split.nsplit;
  if (split.slots > 0) {
    a.part_o = static_cast<float4*>(ws);
    a.part_ml = reinterpret_cast<float2*>(a.part_o + (size_t)split.slots * (2 * kBM * kD / 4));
    x_total = split.split_begin + split.slots;
  }
  dim3 grid(x_total, 1, 1);
  // Launches of one wave overlap their neighbours in the stream, which saves about one K/V step (1.7 us; 100 queries
  // against 16 384 keys, with the merge: 41.1 -> 38.8 us; 256 x 256, 8 heads: 17.0 -> 16.3 us), unless they lose more by
  // it (see overlap_loss: 100 pairs of 50 steps, 83.6 without, 85.2 us with it).  Longer ones lose it in the
  // prologue of their later waves (384 items: 88.0 -> 89.0 us; 256 items: between 1 % faster and 1.6 % slower).
  // Launches with flags or several jobs stay in order: what they wait for may need room on the SMs.
  const int sms = sm_count();
  a.overlap = !has_flags && njobs == 1 && a.job[0].done_flag == nullptr && x_total <= sms;
  if (a.overlap) {
    const FwdJob& J = a.job[0];
    long long steps = 0;   // of the longest item
    for (int s = 0; s < nseg; ++s) {
      long long vis = (J.seg_mask >> s) & 1u ? a.seg_sk[s] : 0;
      if (a.causal) vis = min(vis, (long long)J.q_off + J.Sq - a.seg_koff[s]);
      if (vis > 0) steps += (vis + kBN - 1) / kBN;
    }
    a.overlap = (steps + split.nsplit - 1) / split.nsplit * overlap_loss((double)x_total / sms) <= 1.0;
  }
  const auto kernel = split.slots > 0 || pack_shift > 0 ? attn_fwd_kernel<true> : attn_fwd_kernel<false>;
  if (a.overlap) {
    if (!launch_overlapped("launch attn_fwd_kernel", kernel, grid, kFwdThreads, kFwdSmemBytes, stream, maps, a))
      return MB_E_CUDA;
  } else {
    kernel<<<grid, kFwdThreads, kFwdSmemBytes, stream>>>(maps, a);
    if (!cuda_ok(cudaGetLastError(), "launch attn_fwd_kernel")) return MB_E_CUDA;
  }
  if (split.slots > 0) {
    const FwdJob& J = a.job[0];
    FwdMergeArgs m;
    m.part_o = a.part_o; m.part_ml = a.part_ml;
    m.o = J.o; m.o_sb = J.o_sb; m.o_ss = J.o_ss; m.o_sh = J.o_sh;
    m.lse = J.lse; m.lse_sb = J.lse_sb; m.lse_sh = J.lse_sh;
    m.Sq = J.Sq; m.B = a.B; m.Hq = a.Hq; m.n_pairs = J.n_pairs;
    m.pack_shift = a.pack_shift; m.head_block = a.head_block; m.causal = a.causal;
    m.first_item = split.split_begin; m.nsplit = split.nsplit;
    m.scale = a.scale; m.scale_log2 = a.scale_log2;
    const int rows = min(2 * kBM, J.Sq << a.pack_shift);  // a job shorter than one item has no rows past Sq
    if (!launch_overlapped("launch fwd_split_merge_kernel", fwd_split_merge_kernel,
                           dim3(split.slots / split.nsplit, (rows + kMergeRows - 1) / kMergeRows), 256, 0, stream, m))
      return MB_E_CUDA;
  }
  return MB_SUCCESS;
}

int launch_attn_fwd_multi(const mb_attn_fwd_multi_args* x, cudaStream_t stream) {
  return launch_fwd(x, 0, kWhole, nullptr, stream);
}

// One query shard: the single-job form of the launch above.  With a workspace of attn_fwd_workspace(x) bytes the
// launch may split items over their keys; with less (or none) it runs them whole.
int launch_attn_fwd(const mb_attn_fwd_args* x, void* ws, unsigned long long ws_bytes, cudaStream_t stream) {
  if (x == nullptr) return MB_E_INVALID;
  if (x->nseg < 0 || x->nseg > MB_MAX_SEGMENTS) return MB_E_INVALID;
  if (x->sq < 0) return MB_E_INVALID;
  if (x->sq == 0) {
    if (x->head_dim != kD) return MB_E_UNSUPPORTED;
    if (x->batch <= 0 || x->hq <= 0 || x->hkv <= 0 || x->hq % x->hkv != 0) return MB_E_INVALID;
    return MB_SUCCESS;
  }
  static thread_local mb_attn_fwd_multi_args m;
  memset(&m, 0, sizeof(m));
  m.batch = x->batch; m.hq = x->hq; m.hkv = x->hkv; m.head_dim = x->head_dim;
  m.causal = x->causal; m.softmax_scale = x->softmax_scale;
  m.njobs = 1; m.nseg = x->nseg;
  mb_fwd_job& j = m.job[0];
  j.q = x->q; j.q_stride_b = x->q_stride_b; j.q_stride_s = x->q_stride_s; j.q_stride_h = x->q_stride_h;
  j.o = x->o; j.o_stride_b = x->o_stride_b; j.o_stride_s = x->o_stride_s; j.o_stride_h = x->o_stride_h;
  j.lse = x->lse; j.lse_stride_b = x->lse_stride_b; j.lse_stride_h = x->lse_stride_h;
  j.sq = x->sq; j.q_off = x->q_off;
  for (int s = 0; s < x->nseg; ++s) m.seg[s] = x->seg[s];
  m.status = x->status;
  FwdPlan plan{0, kWhole};
  if (x->batch > 0 && x->hq > 0) {
    plan = plan_fwd(x, ws != nullptr && (reinterpret_cast<uintptr_t>(ws) & 15u) == 0);
    if (plan.split.slots * (unsigned long long)kSlotBytes > ws_bytes) plan = plan_fwd(x, false);
  }
  return launch_fwd(&m, plan.pack_shift, plan.split, ws, stream);
}

}  // namespace mb
