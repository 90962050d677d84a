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
#include "plan.h"

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
  if (tb == 0 && b == 0 && t < 64) P.status[t] = 0;
  if (tb >= P.NB) {
    const int per_word = (64 * M.W + 127) / 128, at = tb - P.NB;
    const int w = at / per_word, c = (at - w * per_word) * 128 + t;
    if (w >= t_words || c >= 64 * M.W) return;
    const int64_t* link_b = M.link + (size_t)b * M.R * M.W + (c >> 6);
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
  __shared__ int warp_cnt[4];
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
  }
  if (t == 0) P.run_cnt[(size_t)b * P.NB + tb] = total;
}

// One thread per (kb, qb, b); the runs of the block's q tile sit in shared memory.  A thread stops at the first proof of a
// partial tile, and looks at four q-runs at a time so that their link words are fetched together: counting every
// combination one by one took 21 us on a 16k pack of 240 grants, whose tiles have ten runs and more a side.
__global__ void __launch_bounds__(128) state_kernel(PlanView P, MaskArgs M, uint8_t* state_out) {
  const int kb = blockIdx.x * blockDim.x + threadIdx.x, qb = blockIdx.y, b = blockIdx.z;
  __shared__ int4 s_runs[kTile];
  const size_t tq = (size_t)b * P.NB + qb;
  const int nq = P.run_cnt[tq];
  if ((int)(blockIdx.x * blockDim.x) <= qb) {
    if ((int)threadIdx.x < nq) s_runs[threadIdx.x] = reinterpret_cast<const int4*>(P.runs + tq * kTile)[threadIdx.x];
  }
  __syncthreads();
  if (kb >= P.NB) return;
  uint8_t st = kSkip;
  const int nvq = min(kTile, P.T - qb * kTile);
  if (kb == qb) {
    st = nvq > 0 ? kPartial : kSkip;
  } else if (kb < qb) {
    const int64_t* link_b = M.link ? M.link + (size_t)b * M.R * M.W : nullptr;
    const int4* kr = reinterpret_cast<const int4*>(P.runs + ((size_t)b * P.NB + kb) * kTile);
    const int nk = P.run_cnt[(size_t)b * P.NB + kb];
    bool some = false, none = nvq < kTile;  // allowed / denied combinations seen; kv tiles below the diagonal are complete
    for (int j = 0; j < nk && !(some && none); ++j) {
      const int4 kj = kr[j];  // start, doc, row, col
      for (int i = 0; i < nq && !(some && none); i += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int4 qi = s_runs[min(i + u, nq - 1)];
          const bool ok = qi.y == kj.y || link_bit(link_b, M.R, M.W, qi.z, kj.w);
          some |= ok;
          none |= !ok;
        }
      }
    }
    st = !some ? kSkip : (none ? kPartial : kFull);
  }
  const size_t at = tq * P.NB + kb;
  P.state[at] = st;
  if (state_out) state_out[at] = st;
}

// One warp per line.  transposed == 0: line = q tile, scan kv tiles; 1: line = kv tile, scan q tiles.
// Writes the merged list used by the kernels and, when given, the separate partial / full lists in the
// BlockMask convention (ascending, entries past the count = -1).
struct ListOutputs {
  int32_t *part_cnt, *part_idx, *full_cnt, *full_idx;
};
// blockIdx.z: 0 lines are q tiles, 1 lines are kv tiles; 2 counts, per pair of adjacent q tiles (2p, 2p+1) -- the forward's
// work items, which share one stream of K/V tiles -- the kv tiles at least one of the two reads.
__global__ void __launch_bounds__(128) lists_kernel(PlanView P, ListOutputs fwd_out, ListOutputs bwd_out) {
  const int transposed = blockIdx.z;
  const int line = blockIdx.x * 4 + (threadIdx.x >> 5), b = blockIdx.y, lane = threadIdx.x & 31;
  if (transposed == 2) {
    const int NP = (P.NB + 1) / 2;
    if (line >= NP) return;
    const uint8_t* s0 = P.state + ((size_t)b * P.NB + 2 * line) * P.NB;
    const uint8_t* s1 = (2 * line + 1 < P.NB) ? s0 + P.NB : s0;
    int n = 0;
    for (int kb = lane; kb <= min(2 * line + 1, P.NB - 1); kb += 32) n += (s0[kb] | s1[kb]) != kSkip;
    for (int sh = 16; sh > 0; sh >>= 1) n += __shfl_xor_sync(0xffffffffu, n, sh);
    if (lane == 0) P.pair_cnt[(size_t)b * NP + line] = n;
    return;
  }
  int32_t* part_cnt = transposed ? bwd_out.part_cnt : fwd_out.part_cnt;
  int32_t* part_idx = transposed ? bwd_out.part_idx : fwd_out.part_idx;
  int32_t* full_cnt = transposed ? bwd_out.full_cnt : fwd_out.full_cnt;
  int32_t* full_idx = transposed ? bwd_out.full_idx : fwd_out.full_idx;
  if (line >= P.NB) return;
  const size_t lb = (size_t)b * P.NB + line;
  int32_t* m_idx = (transposed ? P.bwd_idx : P.fwd_idx) + lb * P.NB;
  int n_m = 0, n_p = 0, n_f = 0;
  for (int c0 = 0; c0 < P.NB; c0 += 32) {
    const int c = c0 + lane;
    uint8_t st = kSkip;
    if (c < P.NB) st = transposed ? P.state[((size_t)b * P.NB + c) * P.NB + line] : P.state[lb * P.NB + c];
    const unsigned bm = __ballot_sync(0xffffffffu, st != kSkip);
    const unsigned bp = __ballot_sync(0xffffffffu, st == kPartial);
    const unsigned bf = __ballot_sync(0xffffffffu, st == kFull);
    const unsigned below = (1u << lane) - 1u;
    if (st != kSkip) m_idx[n_m + __popc(bm & below)] = c | (st == kFull ? (int)kFullBit : 0);
    if (part_idx && st == kPartial) part_idx[lb * P.NB + n_p + __popc(bp & below)] = c;
    if (full_idx && st == kFull) full_idx[lb * P.NB + n_f + __popc(bf & below)] = c;
    n_m += __popc(bm); n_p += __popc(bp); n_f += __popc(bf);
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

// Heaviest-first order inside each batch element: rank by descending count, ties by index.
// which = 0: q tiles by fwd_cnt, 1: kv tiles by bwd_cnt, 2: q-tile pairs by pair_cnt.
__global__ void __launch_bounds__(256) order_kernel(PlanView P, int link_t_rows) {
  const int b = blockIdx.y, which = blockIdx.z;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && b == 0 && which == 0) {  // this is the last launch of the pre-pass: stamp the plan (see plan.h)
    P.status[kStampMagic] = kPlanMagic;
    P.status[kStampB] = P.B;
    P.status[kStampT] = P.T;
    P.status[kLinkTRows] = link_t_rows;
  }
  const int n = which == 2 ? (P.NB + 1) / 2 : P.NB;
  const int32_t* cnt = (which == 2 ? P.pair_cnt : which == 1 ? P.bwd_cnt : P.fwd_cnt) + (size_t)b * n;
  int32_t* order = (which == 2 ? P.pair_order : which == 1 ? P.bwd_order : P.fwd_order) + (size_t)b * n;
  __shared__ int4 s_cnt[256];  // 1024 counts at a time, read by all threads alike
  const int ci = i < n ? cnt[i] : 0;
  int rank = 0;
  for (int j0 = 0; j0 < n; j0 += 1024) {
    __syncthreads();
    for (int j = threadIdx.x; j < 1024; j += blockDim.x) reinterpret_cast<int*>(s_cnt)[j] = j0 + j < n ? cnt[j0 + j] : -1;
    __syncthreads();
    const int m = (min(1024, n - j0) + 3) / 4;  // counts of -1 outrank nobody
    for (int q = 0; q < m; ++q) {
      const int4 c = s_cnt[q];
      const int j = j0 + 4 * q;
      rank += (c.x > ci || (c.x == ci && j < i)) + (c.y > ci || (c.y == ci && j + 1 < i)) + (c.z > ci || (c.z == ci && j + 2 < i)) +
              (c.w > ci || (c.w == ci && j + 3 < i));
    }
  }
  if (i < n) order[rank] = i;
}

// Per-token ids from a sorted table of segments: token t gets ids[j] for bounds[j] <= t < bounds[j + 1], and -1 before
// bounds[0] or from bounds[n_seg] on.  This is the device-side half of what the reference does with one slice
// assignment per grant (cross_doc_mask.py:277-294): the host only works out the few hundred segment boundaries.
__global__ void __launch_bounds__(256) segment_ids_kernel(const int32_t* __restrict__ bounds, const int32_t* __restrict__ ids,
                                                          int n_seg, int T, int32_t* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  int lo = 0, hi = n_seg + 1;  // first boundary > t, by bisection over bounds[0 .. n_seg]
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(bounds + mid) <= t) lo = mid + 1; else hi = mid;
  }
  out[t] = (lo == 0 || lo > n_seg) ? -1 : __ldg(ids + lo - 1);
}

cudaError_t launch_segment_ids(const int32_t* bounds, const int32_t* ids, int n_seg, int T, int32_t* out, cudaStream_t stream) {
  segment_ids_kernel<<<(T + 255) / 256, 256, 0, stream>>>(bounds, ids, n_seg, T, out);
  return cudaGetLastError();
}

// Host entry: fills the plan; optional BlockMask-shaped outputs may be null.
cudaError_t launch_block_map(PlanView P, MaskArgs M, uint8_t* state_out, int32_t* kv_cnt, int32_t* kv_idx,
                             int32_t* full_cnt, int32_t* full_idx, int32_t* q_cnt, int32_t* q_idx, int32_t* full_q_cnt,
                             int32_t* full_q_idx, cudaStream_t stream) {
  if (P.NB == 0 || P.B == 0) return cudaSuccess;
  const bool t = M.link != nullptr && M.R > 0 && M.R <= kLinkTMaxRows && 64 * M.W <= kLinkTMaxCols;
  const int t_words = t ? (M.R + 63) / 64 : 0;
  runs_kernel<<<dim3(P.NB + t_words * ((64 * M.W + 127) / 128), P.B), 128, 0, stream>>>(P, M, t_words);
  state_kernel<<<dim3((P.NB + 127) / 128, P.NB, P.B), 128, 0, stream>>>(P, M, state_out);
  lists_kernel<<<dim3((P.NB + 3) / 4, P.B, 3), 128, 0, stream>>>(P, ListOutputs{kv_cnt, kv_idx, full_cnt, full_idx},
                                                                 ListOutputs{q_cnt, q_idx, full_q_cnt, full_q_idx});
  order_kernel<<<dim3((P.NB + 255) / 256, P.B, 3), 256, 0, stream>>>(P, t ? M.R : 0);
  return cudaGetLastError();
}

}  // namespace ts2ts
