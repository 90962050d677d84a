// Masked attention for ONE new query token per sequence against cached K / V (decoding with KV reuse).
//
// The reference has no such path: its generation loop runs the whole forward over all T tokens for every generated
// token and keeps the last row of the logits (model/generation_loop.py:90-92, model/model.py:214-237;
// GENERATION_FEATURE_SPEC.md:163 lists KV caching as not implemented).  With the keys and values of the earlier
// tokens kept, the attention of the new token is one masked row: out = softmax(scale q K^T + mask row) V with
//     allowed(kv) = kv <= q_pos  and  ( doc_ids[q_pos] == doc_ids[kv]  or  bit(link_bits[row(q_pos)], col(kv)) ),
// the same predicate as the training kernels (cross_doc_mask.py:348-357), evaluated per key; no block plan is needed.
//
// HBM-bound work: every allowed key's K and V row is read once, 4 D bytes per key and head.  One launch, grid
// (cluster size, H, B), 16 warps a block.  The warps of a cluster share one (batch, head): warp w of W takes the groups of
// 32 keys w, w + W, w + 2 W, ..., so that stretches without an allowed key spread over all of them.  It evaluates the mask
// for up to four groups at a time (lane = key), queues the allowed keys in shared memory, and takes them off the queue
// kUnroll at a time per row of lanes (D / 8 lanes hold one row, 16 bytes each), the K and V rows of all of them in flight
// together: masked keys cost no traffic and no lane.  Each row of lanes keeps an online softmax (base 2) of its own; they
// are merged by shuffles inside a warp, through shared memory inside a block and through distributed shared memory inside
// the cluster, so no partial result goes to global memory.
//
// B = 2, H = 16, Tk = 32768, D = 128, 13.9 k allowed keys a sequence (228 MB): two kernels over fixed 128-key tiles with K
// before V took 75 + 41 us (a third of the copy rate; the merge walked 256 partial results one after the other).
#include "launch.cuh"
#include "plan.h"
#include "ptx.cuh"

#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>

namespace ts2ts {

namespace cg = cooperative_groups;

struct DecodeParams {
  const __nv_bfloat16 *q, *k, *v;
  int64_t q_sb, q_sh;              // q [B,H,1,D]: batch and head strides (elements)
  int64_t k_sb, k_sh, k_st, v_sb, v_sh, v_st;
  MaskArgs mask;                   // per-token arrays are [B,Tk]
  const int32_t* q_pos;            // [B] position of the query token in the cache, or nullptr = Tk - 1
  __nv_bfloat16* out;              // [B,H,1,D]
  int64_t o_sb, o_sh;
  float* lse;                      // [B,H]
  int H, Tk;
  float scale_log2;
};

constexpr int kDecWarps = 16, kDecGroups = 4, kUnroll = 4;

__device__ __forceinline__ void row_dot(const uint4& raw, const float (&q)[8], float& acc) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    acc = fmaf(__uint_as_float(w[i] << 16), q[2 * i], acc);
    acc = fmaf(__uint_as_float(w[i] & 0xffff0000u), q[2 * i + 1], acc);
  }
}
__device__ __forceinline__ void row_axpy(const uint4& raw, float p, float (&o)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    o[2 * i] = fmaf(p, __uint_as_float(w[i] << 16), o[2 * i]);
    o[2 * i + 1] = fmaf(p, __uint_as_float(w[i] & 0xffff0000u), o[2 * i + 1]);
  }
}

__device__ __forceinline__ bool may_read(const DecodeParams& p, const int64_t* link_row, int qdoc, int doc, int col) {
  if (doc == qdoc) return true;
  if (link_row == nullptr || col < 0 || col >= 64 * p.mask.W) return false;
  return (static_cast<unsigned long long>(__ldg(link_row + (col >> 6))) >> (col & 63)) & 1ull;
}

// A warp's keys once more, kRows at a time and asking for weights of zero: m, l and o into `r`.  For rows that came out as no
// number: keys without weight (padded slots, underflow, all before a maximum that outweighs them) add nothing, whatever
// their values, but 0 * inf is no number.  Asking at every key of the first pass cost everybody (B = 2, H = 16, Tk = 32768,
// D = 128: 42.1 -> 45.6 us, or 44.1 us with this pass inlined behind it).
template <int D>
__device__ __noinline__ void read_carefully(const DecodeParams& p, int qpos, float* r) {
  constexpr int kLanes = D / 8, kRows = 32 / kLanes;
  const int h = blockIdx.y, b = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t base = (size_t)b * p.Tk;
  const int qdoc = p.mask.doc[base + qpos], row = p.mask.row[base + qpos];
  const int64_t* link_row = p.mask.link != nullptr && row >= 0 && row < p.mask.R ? p.mask.link + ((size_t)b * p.mask.R + row) * p.mask.W : nullptr;
  const int sub = lane / kLanes, at = (lane % kLanes) * 8;
  float q[8], o[8], m = -CUDART_INF_F, l = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    q[i] = __bfloat162float(p.q[(size_t)b * p.q_sb + (size_t)h * p.q_sh + at + i]) * p.scale_log2;
    o[i] = 0.f;
  }
#pragma unroll 1
  for (int g = blockIdx.x * kDecWarps + warp; g < qpos / 32 + 1; g += gridDim.x * kDecWarps) {
    const int kv = g * 32 + lane;
    unsigned keys = __ballot_sync(0xffffffffu, kv <= qpos && may_read(p, link_row, qdoc, p.mask.doc[base + kv], p.mask.col[base + kv]));
#pragma unroll 1
    while (keys) {
      int key = g * 32 + __ffs(keys) - 1;  // of the first row of lanes; rows without a key of their own repeat it
      bool live = sub == 0;
      keys &= keys - 1;
#pragma unroll
      for (int k = 1; k < kRows; ++k) {
        if (sub == k && keys) { key = g * 32 + __ffs(keys) - 1; live = true; }
        keys &= keys - 1;
      }
      const uint4 kr = __ldg(reinterpret_cast<const uint4*>(p.k + (size_t)b * p.k_sb + (size_t)h * p.k_sh + (size_t)key * p.k_st + at));
      const uint4 vr = __ldg(reinterpret_cast<const uint4*>(p.v + (size_t)b * p.v_sb + (size_t)h * p.v_sh + (size_t)key * p.v_st + at));
      float s = 0.f;
      row_dot(kr, q, s);
#pragma unroll
      for (int x = kLanes / 2; x > 0; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
      if (!live) s = -CUDART_INF_F;
      const float mx = fmaxf(m, s), safe = mx == -CUDART_INF_F ? 0.f : mx;
      const float f = fast_exp2(m - safe), w = fast_exp2(s - safe);
      m = mx;
      l = l * f + w;
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = f == 0.f ? 0.f : o[i] * f;
      if (w != 0.f) row_axpy(vr, w, o);
    }
  }
  r[0] = m; r[1] = l;
#pragma unroll
  for (int i = 0; i < 8; ++i) r[2 + i] = o[i];
}

template <int D>
__global__ void __launch_bounds__(kDecWarps * 32, 2) decode_kernel(const __grid_constant__ DecodeParams p) {
  constexpr int kLanes = D / 8;            // lanes that share a row
  constexpr int kRows = 32 / kLanes;       // rows a warp reads at once
  constexpr int kBatch = kRows * kUnroll;  // keys a warp takes off its queue at once
  __shared__ int s_queue[kDecWarps][kDecGroups * 32 + kBatch];
  __shared__ float s_m[kDecWarps], s_l[kDecWarps], s_o[kDecWarps][D];
  __shared__ float s_block[2 + D];         // the block's maximum, sum and unnormalised output row, read by the cluster's first block
  const cg::cluster_group cluster = cg::this_cluster();
  const int h = blockIdx.y, b = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cs = gridDim.x, W = cs * kDecWarps;
  wait_previous();
  const int qpos = p.q_pos ? min(max(p.q_pos[b], 0), p.Tk - 1) : p.Tk - 1;
  const size_t base = (size_t)b * p.Tk;
  const int32_t* docs = p.mask.doc + base;
  const int32_t* cols = p.mask.col + base;
  const int qdoc = docs[qpos];
  const int64_t* link_row = nullptr;
  if (p.mask.link != nullptr) {
    const int row = p.mask.row[base + qpos];
    if (row >= 0 && row < p.mask.R) link_row = p.mask.link + ((size_t)b * p.mask.R + row) * p.mask.W;
  }
  const int sub = lane / kLanes, at = (lane % kLanes) * 8;
  const __nv_bfloat16* kbase = p.k + (size_t)b * p.k_sb + (size_t)h * p.k_sh + at;
  const __nv_bfloat16* vbase = p.v + (size_t)b * p.v_sb + (size_t)h * p.v_sh + at;
  float q[8], o[8];
  {
    const __nv_bfloat16* qrow = p.q + (size_t)b * p.q_sb + (size_t)h * p.q_sh + at;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      q[i] = __bfloat162float(qrow[i]) * p.scale_log2;
      o[i] = 0.f;
    }
  }
  float m = -CUDART_INF_F, l = 0.f;
  int* queue = s_queue[warp];
  int queued = 0;

  // `count` keys off the queue from `from`; slots past the last one repeat it with a score of -inf
  auto take = [&](int from, int count) {
    uint4 kr[kUnroll], vr[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int key = queue[from + min(u * kRows + sub, count - 1)];
      kr[u] = __ldg(reinterpret_cast<const uint4*>(kbase + (size_t)key * p.k_st));
      vr[u] = __ldg(reinterpret_cast<const uint4*>(vbase + (size_t)key * p.v_st));
    }
    float s[kUnroll], mx = m;
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      s[u] = 0.f;
      row_dot(kr[u], q, s[u]);
#pragma unroll
      for (int x = kLanes / 2; x > 0; x >>= 1) s[u] += __shfl_xor_sync(0xffffffffu, s[u], x);
      if (u * kRows + sub >= count) s[u] = -CUDART_INF_F;
      mx = fmaxf(mx, s[u]);
    }
    const float safe = mx == -CUDART_INF_F ? 0.f : mx;
    const float f = fast_exp2(m - safe);  // exp2(-inf) = 0 before the first key
    m = mx;
    l *= f;
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] *= f;
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const float pj = fast_exp2(s[u] - safe);
      l += pj;
      row_axpy(vr[u], pj, o);
    }
  };

  const int n_groups = qpos / 32 + 1;
  for (int g0 = blockIdx.x * kDecWarps + warp; g0 < n_groups; g0 += kDecGroups * W) {
    int doc[kDecGroups], col[kDecGroups];
#pragma unroll
    for (int u = 0; u < kDecGroups; ++u) {
      const int kv = (g0 + u * W) * 32 + lane;
      doc[u] = kv <= qpos ? docs[kv] : 0;
      col[u] = link_row != nullptr && kv <= qpos ? cols[kv] : -1;
    }
#pragma unroll
    for (int u = 0; u < kDecGroups; ++u) {
      const int kv = (g0 + u * W) * 32 + lane;
      bool ok = false;
      if (kv <= qpos) {
        ok = doc[u] == qdoc;
        if (!ok && col[u] >= 0 && col[u] < 64 * p.mask.W)
          ok = (static_cast<unsigned long long>(__ldg(link_row + (col[u] >> 6))) >> (col[u] & 63)) & 1ull;
      }
      const unsigned bal = __ballot_sync(0xffffffffu, ok);
      if (ok) queue[queued + __popc(bal & ((1u << lane) - 1u))] = kv;
      queued += __popc(bal);
    }
    __syncwarp();
    int done = 0;
    for (; queued - done >= kBatch; done += kBatch) take(done, kBatch);
    const int left = queued - done;
    const int kept = lane < left ? queue[done + lane] : 0;
    __syncwarp();
    if (lane < left) queue[lane] = kept;
    queued = left;
    __syncwarp();
  }
  if (queued > 0) take(0, queued);
  bool bad = false;
#pragma unroll
  for (int i = 0; i < 8; ++i) bad = bad || o[i] != o[i];
  if (__any_sync(0xffffffffu, bad)) {
    float r[10];
    read_carefully<D>(p, qpos, r);
    m = r[0]; l = r[1];
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = r[2 + i];
  }

  // rows of lanes -> warp
  float mw = m;
#pragma unroll
  for (int x = kLanes; x < 32; x <<= 1) mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, x));
  const float fw = m == -CUDART_INF_F ? 0.f : fast_exp2(m - mw);
  l *= fw;
#pragma unroll
  for (int i = 0; i < 8; ++i) o[i] = fw == 0.f ? 0.f : o[i] * fw;
#pragma unroll
  for (int x = kLanes; x < 32; x <<= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, x);
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] += __shfl_xor_sync(0xffffffffu, o[i], x);
  }
  if (sub == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) s_o[warp][at + i] = o[i];
  }
  if (lane == 0) { s_m[warp] = mw; s_l[warp] = l; }
  __syncthreads();
  // warps -> block
  const int d = threadIdx.x;
  if (d < D) {
    float mb = s_m[0];
#pragma unroll
    for (int w = 1; w < kDecWarps; ++w) mb = fmaxf(mb, s_m[w]);
    float lb = 0.f, ob = 0.f;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) {
      const float f = s_m[w] == -CUDART_INF_F ? 0.f : fast_exp2(s_m[w] - mb);
      lb = fmaf(f, s_l[w], lb);
      ob = fmaf(f, f == 0.f ? 0.f : s_o[w][d], ob);
    }
    if (d == 0) { s_block[0] = mb; s_block[1] = lb; }
    s_block[2 + d] = ob;
  }
  cluster.sync();
  // blocks -> out
  if (blockIdx.x == 0 && d < D) {
    float mc = -CUDART_INF_F;
    for (int r = 0; r < cs; ++r) mc = fmaxf(mc, *cluster.map_shared_rank(&s_block[0], r));
    float lc = 0.f, oc = 0.f;
    for (int r = 0; r < cs; ++r) {
      const float mr = *cluster.map_shared_rank(&s_block[0], r), lr = *cluster.map_shared_rank(&s_block[1], r);
      const float xr = *cluster.map_shared_rank(&s_block[2 + d], r);
      const float f = mr == -CUDART_INF_F ? 0.f : fast_exp2(mr - mc);
      lc = fmaf(f, lr, lc);
      oc = fmaf(f, f == 0.f ? 0.f : xr, oc);
    }
    p.out[(size_t)b * p.o_sb + (size_t)h * p.o_sh + d] = __float2bfloat16(lc > 0.f ? oc / lc : 0.f);
    if (d == 0) p.lse[(size_t)b * p.H + h] = lc > 0.f ? (mc + log2f(lc)) * 0.6931471805599453f : -CUDART_INF_F;
  }
  cluster.sync();  // the first block has read the others' shared memory
}

// No partial results go through global memory; the argument stays part of the interface.
size_t decode_workspace_bytes(int, int, int, int) { return 256; }

int launch_decode(const void* q, const void* k, const void* v, const int64_t* sq, const int64_t* sk, const int64_t* sv, int B, int H,
                  int Tk, int D, float scale, MaskArgs M, const int32_t* q_pos, void* out, const int64_t* so, float* lse,
                  cudaStream_t stream) {
  DecodeParams p;
  p.q = static_cast<const __nv_bfloat16*>(q); p.k = static_cast<const __nv_bfloat16*>(k); p.v = static_cast<const __nv_bfloat16*>(v);
  p.q_sb = sq[0]; p.q_sh = sq[1];
  p.k_sb = sk[0]; p.k_sh = sk[1]; p.k_st = sk[2];
  p.v_sb = sv[0]; p.v_sh = sv[1]; p.v_st = sv[2];
  p.mask = M; p.q_pos = q_pos;
  p.out = static_cast<__nv_bfloat16*>(out); p.o_sb = so[0]; p.o_sh = so[1];
  p.lse = lse;
  p.H = H; p.Tk = Tk;
  p.scale_log2 = scale * 1.4426950408889634f;
  // Blocks per (batch, head): twice the SM count in all, as long as every warp gets two groups of keys; eight is the
  // largest cluster every part of the chip takes.
  const long long groups = (Tk + 31) / 32;
  int cs = 1;
  while (cs < 8 && (long long)B * H * cs < 2 * 148 && groups >= 2ll * kDecWarps * 2 * cs) cs *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs, H, B);
  cfg.blockDim = dim3(kDecWarps * 32);
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = cs; attrs[0].val.clusterDim.y = 1; attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see launch.cuh
  attrs[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = 2;
  if (D == 128) return cudaLaunchKernelEx(&cfg, decode_kernel<128>, p) == cudaSuccess ? 0 : -141;
  if (D == 64) return cudaLaunchKernelEx(&cfg, decode_kernel<64>, p) == cudaSuccess ? 0 : -141;
  return -142;
}

}  // namespace ts2ts
