// Integer pre-pass: per-token doc ids / row classes / column classes / link bits
// -> 128x128 block map (skip / partial / full), ordered block lists and a
// heaviest-first tile order.  Replaces, in O(tiles x runs) integer work, what the
// reference obtains from torch's create_block_mask by materialising the dense
// T x T mask (called at block_mask_creator.py:132-139, cross_doc_mask.py:359-366;
// block sums at torch/nn/attention/flex_attention.py:1034-1084).
//
// A tile is cut into runs of constant (doc, row class, column class).  For a
// tile pair below the diagonal, with
//   allowed(i, j) = doc_i == doc_j  or  bit(link[row_i], col_j)
// over (q-run i, kv-run j), the pair is skipped when no combination is allowed,
// full when all are and partial as soon as one of each kind is found.
// Tokens past T belong to no run, which reproduces torch's pad-with-False: a
// ragged last tile is never full.  A diagonal pair always holds its own
// diagonal (allowed) and the upper triangle (not allowed), so it is partial.
#include "launch.cuh"
#include "plan.h"
#include "ptx.cuh"

#include <cuda_runtime.h>

namespace ts2ts {

__device__ __forceinline__ bool link_bit(const int64_t* link_b, int R, int W, int row, int col) {
  if (link_b == nullptr || row < 0 || row >= R || col < 0 || col >= 64 * W) return false;
  const unsigned long long w = static_cast<unsigned long long>(link_b[(size_t)row * W + (col >> 6)]);
  return (w >> (col & 63)) & 1ull;
}

// First launch, 128 threads.  Blocks (tile, b) with tile < NB cut a tile into runs; the blocks after them transpose the
// link bits (if `t_words` > 0), one thread per (64 row classes, column class): both only need the inputs, and a launch
// of its own cost more than either.  The first block clears the status words.
__global__ void __launch_bounds__(128) runs_kernel(PlanView P, MaskArgs M, int t_words) {
  const int tb = blockIdx.x, b = blockIdx.y, t = threadIdx.x;
  wait_previous();
  let_next_start();
  if (tb == 0 && b == 0 && t < 64) P.status[t] = 0;
  if (tb >= P.NB) {
    const int per_word = (64 * M.W + 127) / 128, at = tb - P.NB;
    const int w = at / per_word, c = (at - w * per_word) * 128 + t;
    if (w >= t_words || c >= 64 * M.W) return;
    const int64_t* link_b = settled(M.link) + (size_t)b * M.R * M.W + (c >> 6);
    const int r0 = 64 * w, n = min(64, M.R - r0);
    unsigned long long out = 0ull;
#pragma unroll 8
    for (int r = 0; r < n; ++r) out |= ((static_cast<unsigned long long>(__ldg(link_b + (size_t)(r0 + r) * M.W)) >> (c & 63)) & 1ull) << r;
    P.link_t[((size_t)b * kLinkTMaxCols + c) * kLinkTWords + w] = out;
    return;
  }
  const int pos = tb * kTile + t;
  const bool valid = pos < P.T;
  const size_t base = (size_t)b * P.T;
  int d = 0, r = 0, c = 0;
  bool flag = false;
  if (valid) {
    d = M.doc[base + pos]; r = M.row[base + pos]; c = M.col[base + pos];
    if (t == 0) flag = true;
    else flag = d != M.doc[base + pos - 1] || r != M.row[base + pos - 1] || c != M.col[base + pos - 1];
  }
  __shared__ int warp_cnt[4], s_start[kMaskRuns + 1];
  if (t <= kMaskRuns) s_start[t] = min(kTile, P.T - tb * kTile);
  const unsigned bal = __ballot_sync(0xffffffffu, flag);
  const int lane = t & 31, w = t >> 5;
  if (lane == 0) warp_cnt[w] = __popc(bal);
  __syncthreads();
  int off = 0;
  for (int i = 0; i < w; ++i) off += warp_cnt[i];
  const int total = warp_cnt[0] + warp_cnt[1] + warp_cnt[2] + warp_cnt[3];
  if (flag) {
    const int idx = off + __popc(bal & ((1u << lane) - 1u));
    Run run; run.start = t; run.doc = d; run.row = r; run.col = c;
    P.runs[((size_t)b * P.NB + tb) * kTile + idx] = run;
    if (idx <= kMaskRuns) s_start[idx] = t;
  }
  if (t == 0) P.run_cnt[(size_t)b * P.NB + tb] = total;
  __syncthreads();
  if (t < kMaskRuns) {  // runs past the last one come out empty
    uint32_t lo[4], hi[4];
    prefix_mask(s_start[t], lo);
    prefix_mask(s_start[t + 1], hi);
    P.run_mask[((size_t)b * P.NB + tb) * kMaskRuns + t] = make_uint4(hi[0] & ~lo[0], hi[1] & ~lo[1], hi[2] & ~lo[2], hi[3] & ~lo[3]);
  }
}

// State of every tile pair and the masks of the partial ones (see kMaskRuns in plan.h).  A block walks 32 pairs of one q
// tile; the runs of the q tile, and the documents, column classes and token masks of the first eight runs of each kv tile
// sit in shared memory.  Eight lanes share a pair: lane i tests q run i against the kv runs one by one and collects its
// column mask; votes then tell it, as the lane of kv run i, which q runs may read that one.  The kernel is bound by the
// instructions it issues (18 us at B = 2, T = 32768 with sixteen lanes a pair and the kv runs passed round by shuffles,
// 20 us with dependent loads instead).  Tiles of more than eight runs take the loop over the run lists.
constexpr int kStateKb = 32;
__device__ __forceinline__ void add_run(uint32_t (&bits)[4], int start, int end) {
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    const int lo = max(start - 32 * w, 0), hi = min(end - 32 * w, 32);
    if (hi > lo) bits[w] |= (hi - lo == 32 ? 0xffffffffu : ((1u << (hi - lo)) - 1u)) << lo;
  }
}
__global__ void __launch_bounds__(128) state_kernel(PlanView P, MaskArgs M, uint8_t* state_out) {
  const int kb0 = blockIdx.x * kStateKb, qb = blockIdx.y, b = blockIdx.z;
  const size_t tq = (size_t)b * P.NB + qb;
  after_previous();
  if (kb0 > qb) {  // above the diagonal
    const int kb = kb0 + threadIdx.x;
    if (threadIdx.x < kStateKb && kb < P.NB) {
      P.state[tq * P.NB + kb] = 0u;
      if (state_out) state_out[tq * P.NB + kb] = kSkip;
    }
    return;
  }
  __shared__ int4 s_runs[kTile];  // start, doc, row class, column class
  __shared__ uint4 s_qmask[kMaskRuns], s_kmask[kStateKb][kMaskRuns + 1];  // + 1: the four pairs of a warp fall on different banks
  __shared__ int2 s_krun[kStateKb][kMaskRuns + 1];                        // doc, column class
  __shared__ int s_nk[kStateKb];
  const size_t tk0 = (size_t)b * P.NB + kb0;
  const int n_kb = min(kStateKb, min(P.NB - kb0, qb + 1 - kb0));
  const int nq = min(P.run_cnt[tq], kTile);
  if (threadIdx.x < kMaskRuns) s_qmask[threadIdx.x] = P.run_mask[tq * kMaskRuns + threadIdx.x];
  if ((int)threadIdx.x < n_kb) s_nk[threadIdx.x] = min(P.run_cnt[tk0 + threadIdx.x], kTile);
#pragma unroll
  for (int i = threadIdx.x; i < kStateKb * kMaskRuns; i += 128) {
    const int k = i / kMaskRuns, r = i % kMaskRuns;
    if (k < n_kb) {
      const int4 run = reinterpret_cast<const int4*>(P.runs + (tk0 + k) * kTile)[r];
      s_krun[k][r] = make_int2(run.y, run.w);
      s_kmask[k][r] = P.run_mask[(tk0 + k) * kMaskRuns + r];
    }
  }
  if ((int)threadIdx.x < nq) s_runs[threadIdx.x] = reinterpret_cast<const int4*>(P.runs + tq * kTile)[threadIdx.x];
  __syncthreads();
  const int64_t* link_b = M.link ? M.link + (size_t)b * M.R * M.W : nullptr;
  const int lane = threadIdx.x & 31, mine = lane & 7;
  const int nvq = min(kTile, P.T - qb * kTile);
  const size_t pairs = (size_t)b * ((size_t)P.NB * (P.NB + 1) / 2);
  const int4 q_run = s_runs[min(mine, nq - 1)];
  unsigned long long lw[4] = {0ull, 0ull, 0ull, 0ull};  // the first four link words of this lane's q run
  if (link_b != nullptr && q_run.z >= 0 && q_run.z < M.R) {
#pragma unroll
    for (int w = 0; w < 4; ++w)
      if (w < M.W) lw[w] = static_cast<unsigned long long>(__ldg(link_b + (size_t)q_run.z * M.W + w));
  }
#pragma unroll 1
  for (int k = threadIdx.x >> 3; k < kStateKb; k += 16) {
    const int kb = kb0 + k;
    const bool below = k < n_kb;
    const int nk = below ? s_nk[k] : 0;
    bool some = false, none = false;
    uint32_t qbits[4] = {0u, 0u, 0u, 0u}, kbits[4] = {0u, 0u, 0u, 0u};  // mask of q run `mine` over keys, of kv run `mine` over query rows
    const int most = __reduce_max_sync(0xffffffffu, nk);
    if (nq <= kMaskRuns && most <= kMaskRuns) {
      unsigned readers = 0;  // the q runs that may read kv run `mine`
      const bool q_live = mine < nq;
#pragma unroll 1
      for (int j = 0; j < most; ++j) {
        const int2 kr = s_krun[k][j];
        const uint4 km = s_kmask[k][j];
        const bool valid = q_live && j < nk;
        bool ok = kr.x == q_run.y;
        if (!ok && kr.y >= 0) {
          if (kr.y < 256) {
            const int wi = kr.y >> 6;
            ok = ((wi == 0 ? lw[0] : wi == 1 ? lw[1] : wi == 2 ? lw[2] : lw[3]) >> (kr.y & 63)) & 1ull;
          } else if (valid) {
            ok = link_bit(link_b, M.R, M.W, q_run.z, kr.y);
          }
        }
        ok = ok && valid;
        some |= ok;
        none |= valid && !ok;
        if (ok) { qbits[0] |= km.x; qbits[1] |= km.y; qbits[2] |= km.z; qbits[3] |= km.w; }
        const unsigned bal = __ballot_sync(0xffffffffu, ok);
        if (mine == j) readers = bal >> (lane & 24);
      }
      for (int i = 0; i < nq; ++i)
        if ((readers >> i) & 1u) {
          const uint4 q = s_qmask[i];
          kbits[0] |= q.x; kbits[1] |= q.y; kbits[2] |= q.z; kbits[3] |= q.w;
        }
    } else {
      const int4* kr = reinterpret_cast<const int4*>(P.runs + (tk0 + (below ? k : 0)) * kTile);
      const int nvk = min(kTile, P.T - kb * kTile);
#pragma unroll 1
      for (int i = mine; i < (below ? nq : 0); i += 8)
#pragma unroll 1
        for (int j = 0; j < nk; ++j) {
          const int4 me = s_runs[i], other = kr[j];
          const bool ok = me.y == other.y || link_bit(link_b, M.R, M.W, me.z, other.w);
          some |= ok;
          none |= !ok;
          if (ok && i < kMaskRuns) add_run(qbits, other.x, j + 1 < nk ? kr[j + 1].x : nvk);
        }
      if (below && mine < nk) {
        const int4 me = kr[mine];
#pragma unroll 1
        for (int i = 0; i < nq; ++i)
          if (me.y == s_runs[i].y || link_bit(link_b, M.R, M.W, s_runs[i].z, me.w)) add_run(kbits, s_runs[i].x, i + 1 < nq ? s_runs[i + 1].x : nvq);
      }
    }
    const unsigned group = 0xffu << (lane & 24);
    const bool any_some = (__ballot_sync(0xffffffffu, some) & group) != 0u, any_none = (__ballot_sync(0xffffffffu, none) & group) != 0u;
    // a ragged q tile is never full, a diagonal pair always partial; kv tiles below the diagonal are complete
    uint8_t st = !below || !any_some ? kSkip : (any_none || nvq < kTile ? kPartial : kFull);
    if (kb == qb) st = kPartial;
    // a partial pair's stretches that some key's mask has a row of: one reduction for the four pairs of the warp, four bits each
    uint32_t live = 0u;
    if (__any_sync(0xffffffffu, st == kPartial)) {
#pragma unroll
      for (int w = 0; w < kStretches; ++w) live |= kbits[w] != 0u ? 1u << w : 0u;
      const int at = (lane & 24) >> 1;
      live = (__reduce_or_sync(0xffffffffu, (mine < nk ? live : 0u) << at) >> at) & kStateLive;
      if (st == kPartial && nk > kMaskRuns) live = (1u << ((nvq + kStretch - 1) / kStretch)) - 1u;  // keys of later runs have no mask: any row may be theirs
    }
    if (mine == 0 && kb < P.NB) {
      P.state[tq * P.NB + kb] = st == kFull ? kStateFull | kStateLive : live;
      if (state_out) state_out[tq * P.NB + kb] = st;
    }
    if (st == kPartial && P.q_mask != nullptr) {
      const size_t pair = pairs + mask_pair(qb, kb);
      if (mine < nq) P.q_mask[pair * kMaskRuns + mine] = make_uint4(qbits[0], qbits[1], qbits[2], qbits[3]);
      if (mine < nk) {
#pragma unroll
        for (int w = 0; w < kStretches; ++w) P.kv_mask[(pair * kStretches + w) * kMaskRuns + mine] = kbits[w];
      }
    }
  }
}

// One warp per line.  A line is a q tile, whose kv tiles are scanned, or (transposed) a kv tile, whose q tiles are.
// Writes the merged list used by the kernels and, when given, the separate partial / full lists in the
// BlockMask convention (ascending, entries past the count = -1).
struct ListOutputs {
  int32_t *part_cnt, *part_idx, *full_cnt, *full_idx;
};
// The line of a kv tile where the backward's table exists (at most kMaskMaxTiles tiles), by kWarps warps: the separate lists as above, and the
// stretches of the q tiles in the order of PlanLayout::bwd_sub.  A warp owns its share of the line: it loads its states at once, counts
// them, and with the counts of the warps before it and of all every entry has its place.  (Always one warp a line: B = 2, T = 32768 linked
// 5.8 us for the launch, of which the sweep over the line 0.7 and its stores 0.8; four warps 4.6; without the table 4.2.  Four sequences
// of 4096: the whole pre-pass 12.8 us with one warp a line and 14.5 with four, 16384 16.0 and 15.3.)
constexpr int kOneWarpTiles = 64;
template <int kWarps>
__device__ __forceinline__ void stretch_line(const PlanView& P, const ListOutputs& out, int b, int line) {
  constexpr int kMost = 4;  // tiles of a lane
  static_assert(kMost * 32 * 4 == kMaskMaxTiles && kMost * 32 >= kOneWarpTiles, "");
  const int warp = threadIdx.x / 32 % kWarps, lane = threadIdx.x & 31;
  const int sweeps = (P.NB - line + 32 * kWarps - 1) / (32 * kWarps), c0 = line + warp * 32 * sweeps + lane;
  const uint8_t* column = P.state + ((size_t)b * P.NB + c0) * P.NB + line;
  uint32_t sts[kMost];
#pragma unroll
  for (int u = 0; u < kMost; ++u) sts[u] = u < sweeps && c0 + 32 * u < P.NB ? column[(size_t)(32 * u) * P.NB] : 0u;
  // full tiles and all that are not skipped; tiles with four live stretches, which the full ones are too, and the stretches of the others
  uint32_t tiles = 0u, subs = 0u;
#pragma unroll
  for (int u = 0; u < kMost; ++u) {
    const uint32_t live = sts[u] & kStateLive;
    tiles += (sts[u] & kStateFull ? 1u << 16 : 0u) + (live != 0u ? 1u : 0u);
    subs += live == kStateLive ? 1u << 16 : __popc(live);
  }
  tiles = __reduce_add_sync(0xffffffffu, tiles);
  subs = __reduce_add_sync(0xffffffffu, subs);
  uint32_t tiles_to = 0u, subs_to = 0u;
  if (kWarps > 1) {
    __shared__ uint2 s_counts[kWarps];
    if (lane == 0) s_counts[warp] = make_uint2(tiles, subs);
    __syncthreads();
    tiles = subs = 0u;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const uint2 n = s_counts[w];
      if (w < warp) { tiles_to += n.x; subs_to += n.y; }
      tiles += n.x; subs += n.y;
    }
  }
  const int n_full = tiles >> 16, n_part = (tiles & 0xffffu) - n_full, n_whole = subs >> 16, n_subs = kStretches * n_whole + (subs & 0xffffu);
  int at_full = tiles_to >> 16, at_part = (tiles_to & 0xffffu) - at_full;
  int at_live = n_full + (subs_to >> 16) - at_full, at_rest = kStretches * n_whole + (subs_to & 0xffffu);
  const size_t lb = (size_t)b * P.NB + line;
  const unsigned below = (1u << lane) - 1u;
  uint16_t* sub = P.bwd_sub + ((size_t)b * sub_line(P.NB, P.NB) + sub_line(P.NB, line)) * kStretches;
#pragma unroll
  for (int u = 0; u < kMost; ++u) {
    const uint32_t st = sts[u], qb = c0 + 32 * u, first = kStretches * qb;
    const bool full = (st & kStateFull) != 0u, whole = (st & kStateLive) == kStateLive;
    const unsigned b_any = __ballot_sync(0xffffffffu, st != 0u), b_full = __ballot_sync(0xffffffffu, full), b_whole = __ballot_sync(0xffffffffu, whole);
    if (b_any == 0u) continue;
    if (whole) {
      const uint32_t lo = (first | (first + 1u) << 16) | (full ? kStretchFull | kStretchFull << 16 : 0u);
      const int at = full ? at_full + __popc(b_full & below) : at_live + __popc(b_whole & ~b_full & below);
      *reinterpret_cast<uint2*>(sub + kStretches * at) = make_uint2(lo, lo + 0x20002u);
    }
    if (b_any != b_whole) {
      const uint32_t live = whole ? 0u : st & kStateLive;
      int at = at_rest;
#pragma unroll
      for (int w = 0; w < kStretches; ++w) {
        const unsigned bal = __ballot_sync(0xffffffffu, (live >> w) & 1u);
        at += __popc(bal & below);
        at_rest += __popc(bal);
      }
#pragma unroll
      for (int w = 0; w < kStretches; ++w)
        if ((live >> w) & 1u) sub[at++] = first + w;
    }
    if (out.part_idx && st != 0u && !full) out.part_idx[lb * P.NB + at_part + __popc(b_any & ~b_full & below)] = qb;
    if (out.full_idx && full) out.full_idx[lb * P.NB + at_full + __popc(b_full & below)] = qb;
    at_part += __popc(b_any & ~b_full);
    at_full += __popc(b_full);
    at_live += __popc(b_whole & ~b_full);
  }
  const int t = threadIdx.x % (32 * kWarps), n_vt = (n_subs + kStretches - 1) / kStretches;
  if (t < kStretches * n_vt - n_subs) sub[n_subs + t] = kStretches * P.NB;
  if (out.part_idx) for (int c = n_part + t; c < P.NB; c += 32 * kWarps) out.part_idx[lb * P.NB + c] = -1;
  if (out.full_idx) for (int c = n_full + t; c < P.NB; c += 32 * kWarps) out.full_idx[lb * P.NB + c] = -1;
  if (t == 0) {
    P.bwd_cnt[lb] = n_part + n_full;
    P.bwd_tiles[lb] = n_vt;
    if (out.part_cnt) out.part_cnt[lb] = n_part;
    if (out.full_cnt) out.full_cnt[lb] = n_full;
  }
}

// Blocks of a batch element: first the lines of kv tiles, one each where four warps share them and four otherwise, then four lines of q tiles each; the rest count, per pair of adjacent q tiles (2p, 2p+1) -- the forward's work items, which share one stream of K/V
// tiles -- the kv tiles at least one of the two reads, four pairs each.
__host__ __device__ inline bool kv_line_a_block(const PlanView& P) { return P.bwd_sub != nullptr && P.NB > kOneWarpTiles; }
static int lists_blocks(const PlanView& P) {
  const int four = (P.NB + 3) / 4;
  return (kv_line_a_block(P) ? P.NB : four) + four + ((P.NB + 1) / 2 + 3) / 4;
}
__global__ void __launch_bounds__(128) lists_kernel(PlanView P, ListOutputs fwd_out, ListOutputs bwd_out) {
  const int four = (P.NB + 3) / 4, kv_blocks = kv_line_a_block(P) ? P.NB : four;
  const bool transposed = (int)blockIdx.x < kv_blocks, pairs = (int)blockIdx.x >= kv_blocks + four;
  const int b = blockIdx.y, lane = threadIdx.x & 31;
  const int line = (blockIdx.x - (transposed ? 0 : pairs ? kv_blocks + four : kv_blocks)) * 4 + (threadIdx.x >> 5);
  after_previous();
  if (transposed && kv_line_a_block(P)) {
    stretch_line<4>(P, bwd_out, b, blockIdx.x);
    return;
  }
  if (pairs) {
    const int NP = (P.NB + 1) / 2;
    if (line >= NP) return;
    const uint8_t* s0 = P.state + ((size_t)b * P.NB + 2 * line) * P.NB;
    const uint8_t* s1 = (2 * line + 1 < P.NB) ? s0 + P.NB : s0;
    int n = 0;
#pragma unroll 8
    for (int kb = lane; kb <= min(2 * line + 1, P.NB - 1); kb += 32) n += (s0[kb] | s1[kb]) != 0;
    for (int sh = 16; sh > 0; sh >>= 1) n += __shfl_xor_sync(0xffffffffu, n, sh);
    if (lane == 0) P.pair_cnt[(size_t)b * NP + line] = n;
    return;
  }
  int32_t* part_cnt = transposed ? bwd_out.part_cnt : fwd_out.part_cnt;
  int32_t* part_idx = transposed ? bwd_out.part_idx : fwd_out.part_idx;
  int32_t* full_cnt = transposed ? bwd_out.full_cnt : fwd_out.full_cnt;
  int32_t* full_idx = transposed ? bwd_out.full_idx : fwd_out.full_idx;
  if (line >= P.NB) return;
  if (transposed && P.bwd_sub != nullptr) {
    stretch_line<1>(P, bwd_out, b, line);
    return;
  }
  const size_t lb = (size_t)b * P.NB + line;
  int32_t* m_idx = (transposed ? P.bwd_idx : P.fwd_idx) + lb * P.NB;
  int n_m = 0, n_p = 0, n_f = 0;
  constexpr int kAhead = 8;  // states a lane loads before it counts the first: the loads are what a line waits for
  for (int c0 = 0; c0 < P.NB; c0 += 32 * kAhead) {
    uint8_t sts[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int c = c0 + 32 * u + lane;
      sts[u] = 0;
      if (c < P.NB) sts[u] = transposed ? P.state[((size_t)b * P.NB + c) * P.NB + line] : P.state[lb * P.NB + c];
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int c = c0 + 32 * u + lane;
      const uint8_t st = sts[u] == 0 ? kSkip : (sts[u] & kStateFull) ? kFull : kPartial;
      const unsigned bm = __ballot_sync(0xffffffffu, st != kSkip);
      const unsigned bp = __ballot_sync(0xffffffffu, st == kPartial);
      const unsigned bf = __ballot_sync(0xffffffffu, st == kFull);
      const unsigned below = (1u << lane) - 1u;
      if (st != kSkip) m_idx[n_m + __popc(bm & below)] = c | (st == kFull ? (int)kFullBit : 0);
      if (part_idx && st == kPartial) part_idx[lb * P.NB + n_p + __popc(bp & below)] = c;
      if (full_idx && st == kFull) full_idx[lb * P.NB + n_f + __popc(bf & below)] = c;
      n_m += __popc(bm); n_p += __popc(bp); n_f += __popc(bf);
    }
  }
  for (int c = n_m + lane; c < P.NB; c += 32) m_idx[c] = -1;
  if (part_idx) for (int c = n_p + lane; c < P.NB; c += 32) part_idx[lb * P.NB + c] = -1;
  if (full_idx) for (int c = n_f + lane; c < P.NB; c += 32) full_idx[lb * P.NB + c] = -1;
  if (lane == 0) {
    (transposed ? P.bwd_cnt : P.fwd_cnt)[lb] = n_m;
    if (part_cnt) part_cnt[lb] = n_p;
    if (full_cnt) full_cnt[lb] = n_f;
  }
}

// Heaviest-first order inside each batch element: rank by descending count, ties by index.  Eight lanes share a tile and
// compare its count with an eighth of the others each.
// which = 0: q tiles by fwd_cnt, 1: kv tiles by the query tiles the backward walks for them, 2: q-tile pairs by pair_cnt.
constexpr int kOrderLanes = 8, kOrderTiles = 256 / kOrderLanes;
__global__ void __launch_bounds__(256) order_kernel(PlanView P, int link_t_rows) {
  const int b = blockIdx.y, which = blockIdx.z, sub = threadIdx.x % kOrderLanes;
  const int i = blockIdx.x * kOrderTiles + threadIdx.x / kOrderLanes;
  after_previous();
  if (blockIdx.x == 0 && threadIdx.x == 0 && b == 0 && which == 0) {  // this is the last launch of the pre-pass: stamp the plan (see plan.h)
    P.status[kStampMagic] = kPlanMagic;
    P.status[kStampB] = P.B;
    P.status[kStampT] = P.T;
    P.status[kLinkTRows] = link_t_rows;
  }
  const int n = which == 2 ? (P.NB + 1) / 2 : P.NB;
  if ((int)blockIdx.x * kOrderTiles >= n) return;
  const int32_t* cnt = (which == 2 ? P.pair_cnt : which == 0 ? P.fwd_cnt : P.bwd_sub != nullptr ? P.bwd_tiles : P.bwd_cnt) + (size_t)b * n;
  int32_t* order = (which == 2 ? P.pair_order : which == 1 ? P.bwd_order : P.fwd_order) + (size_t)b * n;
  __shared__ int4 s_cnt[256];  // 1024 counts at a time
  const int ci = i < n ? cnt[i] : 0;
  if (which == 0) {  // what the forward chooses its work items by; the adds are on their way while the tiles are ranked
    const int longest = __reduce_max_sync(0xffffffffu, ci), sum = __reduce_add_sync(0xffffffffu, sub == 0 ? ci : 0);
    if (threadIdx.x % 32 == 0) {
      atomicMax(&P.status[kLongestList], longest);
      atomicAdd(&P.status[kAllLists], sum);
    }
  }
  int rank = 0;
  for (int j0 = 0; j0 < n; j0 += 1024) {
    __syncthreads();
    for (int j = threadIdx.x; j < 1024; j += blockDim.x) reinterpret_cast<int*>(s_cnt)[j] = j0 + j < n ? cnt[j0 + j] : -1;
    __syncthreads();
    const int m = (min(1024, n - j0) + 3) / 4;  // counts of -1 outrank nobody
#pragma unroll 4
    for (int q = sub; q < m; q += kOrderLanes) {
      const int4 c = s_cnt[q];
      const int j = j0 + 4 * q;
      rank += (c.x > ci || (c.x == ci && j < i)) + (c.y > ci || (c.y == ci && j + 1 < i)) + (c.z > ci || (c.z == ci && j + 2 < i)) +
              (c.w > ci || (c.w == ci && j + 3 < i));
    }
  }
#pragma unroll
  for (int x = kOrderLanes / 2; x > 0; x >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, x);
  if (i < n && sub == 0) order[rank] = i;
}

// Per-token ids from a sorted table of segments: token t gets ids[j] for bounds[j] <= t < bounds[j + 1], and -1 before
// bounds[0] or from bounds[n_seg] on.  This is the device-side half of what the reference does with one slice
// assignment per grant (cross_doc_mask.py:277-294): the host only works out the few hundred segment boundaries.
__global__ void __launch_bounds__(256) segment_ids_kernel(const int32_t* __restrict__ bounds, const int32_t* __restrict__ ids,
                                                          int n_seg, int T, int32_t* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  wait_previous();
  bounds = settled(bounds);
  ids = settled(ids);
  if (t >= T) return;
  int lo = 0, hi = n_seg + 1;  // first boundary > t, by bisection over bounds[0 .. n_seg]
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(bounds + mid) <= t) lo = mid + 1; else hi = mid;
  }
  out[t] = (lo == 0 || lo > n_seg) ? -1 : __ldg(ids + lo - 1);
}

cudaError_t launch_segment_ids(const int32_t* bounds, const int32_t* ids, int n_seg, int T, int32_t* out, cudaStream_t stream) {
  return launch_after(segment_ids_kernel, dim3((T + 255) / 256), 256, 0, stream, bounds, ids, n_seg, T, out);
}

// The four launches depend on one another and take a few microseconds each, so each starts while the one before still runs
// (launch.cuh): with the lists' loads ahead and the shared ranking 29.0 -> 24.3-25.8 us a call at B = 2, T = 32768 with explicit lists.
// Without them, linked, us: 4096 11.4, 16384 15.1, 32768 19.4, two of them 22.9, four 31.1, 65536 29.6.  What the backward's gathered tiles need of it
// (masks by stretch and live stretches in `state`, their lines in `lists`) is 0 to 2 of that.
// Host entry: fills the plan; optional BlockMask-shaped outputs may be null.
cudaError_t launch_block_map(PlanView P, MaskArgs M, uint8_t* state_out, int32_t* kv_cnt, int32_t* kv_idx,
                             int32_t* full_cnt, int32_t* full_idx, int32_t* q_cnt, int32_t* q_idx, int32_t* full_q_cnt,
                             int32_t* full_q_idx, cudaStream_t stream) {
  if (P.NB == 0 || P.B == 0) return cudaSuccess;
  const bool t = M.link != nullptr && M.R > 0 && M.R <= kLinkTMaxRows && 64 * M.W <= kLinkTMaxCols;
  const int t_words = t ? (M.R + 63) / 64 : 0;
  cudaError_t e = launch_after(runs_kernel, dim3(P.NB + t_words * ((64 * M.W + 127) / 128), P.B), 128, 0, stream, P, M, t_words);
  if (e == cudaSuccess) e = launch_after(state_kernel, dim3((P.NB + kStateKb - 1) / kStateKb, P.NB, P.B), 128, 0, stream, P, M, state_out);
  if (e == cudaSuccess)
    e = launch_after(lists_kernel, dim3(lists_blocks(P), P.B), 128, 0, stream, P, ListOutputs{kv_cnt, kv_idx, full_cnt, full_idx},
                     ListOutputs{q_cnt, q_idx, full_q_cnt, full_q_idx});
  if (e == cudaSuccess) e = launch_after(order_kernel, dim3((P.NB + kOrderTiles - 1) / kOrderTiles, P.B, 3), 256, 0, stream, P, t ? M.R : 0);
  const cudaError_t last = cudaGetLastError();
  return e != cudaSuccess ? e : last;
}

}  // namespace ts2ts
