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
// (cluster size, H, B), 16 warps a block.  The blocks of a cluster share one (batch, head) and take its groups of 32 keys in turn.
// A block works in rounds of up to 128 groups (one round for 4096 keys a block): its warps evaluate the mask, lane = key, and write the
// allowed keys into one queue in shared memory, in order; then they take them off it in turn,
// kUnroll keys at a time per row of lanes (D / 8 lanes hold one row, 16 bytes each), the K and V rows of all of them in flight
// together: masked keys cost no traffic and no lane, and a document's keys, which lie together, are every warp's work.  Each row of lanes keeps an online
// softmax (base 2) of its own; they are merged by shuffles inside a warp, through shared memory inside a block and through the first block's shared
// memory inside the cluster, so no partial result goes to global memory.
//
// Warps that took the keys of their own groups waited for the one with most of them (GPU time alone, us, own groups -> one queue: linked 2 x 32768, H = 16,
// D = 128, 8.3 k allowed keys 36.7 -> 30.3 (21 at the copy rate); 16 x 8192, H = 16, D = 128 45.2 -> 38.5; 20000, H = 16, D = 64 13.7 -> 12.0; all keys allowed, 2 x 32768,
// 84.3 -> 85.6).  Up to 64 groups a block the queue's two barriers cost more than that (own | one: eight of 1111, H = 12, D = 64 6.2 | 8.0; 4 x 4590 7.2 | 9.8; at the
// line 8 x 1852, H = 8, D = 128 8.1 | 9.9, all keys of 16 x 2048 46.5 | 51.9), and warps keep their own.  Before the merge went through the first block's memory these
// were 7.2, 8.5, 9.1 and 50.3.
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

constexpr int kDecWarps = 16, kDecGroups = 8, kDecAtOnce = 4, kUnroll = 4, kDecCluster = 8;  // kDecCluster: the largest cluster that every part of the chip takes

// Arrival publishes what the block has written, the other blocks' shared memory included.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

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

// A block's keys once more, a warp's share in groups, kRows at a time and asking for weights of zero: m, l and o into `r`.  For blocks in which a row came out
// as no number: keys without weight (padded slots, underflow, all before a maximum that outweighs them) add nothing, whatever
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
  for (int g = warp * gridDim.x + blockIdx.x; g < qpos / 32 + 1; g += gridDim.x * kDecWarps) {
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

// kQueue: the warps of a block share one queue.  Otherwise each has at most kDecAtOnce groups and takes its own keys.
// kPerSm: blocks an SM is to hold, which sets the registers; with two, 64 a thread, the loads of a batch wait for one another.
template <int D, bool kQueue, int kPerSm>
__global__ void __launch_bounds__(kDecWarps * 32, kPerSm) decode_kernel(const __grid_constant__ DecodeParams p) {
  constexpr int kLanes = D / 8;            // lanes that share a row
  constexpr int kRows = 32 / kLanes;       // rows a warp reads at once
  constexpr int kBatch = kRows * kUnroll;  // keys a warp takes off its queue at once
  constexpr int kGroups = kQueue ? kDecGroups : kDecAtOnce;  // of a warp in a round
  __shared__ int s_queue[kDecWarps * kGroups * 32];
  __shared__ __align__(16) int s_count[kDecWarps * kGroups];
  __shared__ float s_m[kDecWarps], s_l[kDecWarps], s_o[kDecWarps][D];
  __shared__ float s_part[kDecCluster][2 + D];  // in the cluster's first block: every block's maximum, sum and unnormalised output row
  const cg::cluster_group cluster = cg::this_cluster();
  const int h = blockIdx.y, b = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cs = gridDim.x;
  cluster_arrive();  // each block is there before another one writes into its shared memory
  wait_previous();
  const size_t base = (size_t)b * p.Tk;
  const int32_t* docs = p.mask.doc + base;
  const int32_t* cols = p.mask.col + base;
  // Group u of this warp in the round that starts at the block's group `first`.
  auto group_at = [&](int first, int u) { return (first + u * kDecWarps + warp) * cs + blockIdx.x; };
  // The mask inputs of kDecAtOnce groups; tokens past the query are loaded too, and not looked at.
  int doc[kDecAtOnce], col[kDecAtOnce];
  auto fetch = [&](int first) {
#pragma unroll
    for (int u = 0; u < kDecAtOnce; ++u) {
      const int kv = group_at(first, u) * 32 + lane;
      doc[u] = kv < p.Tk ? ld_nc_i32_here(docs + kv) : 0;
      col[u] = p.mask.link != nullptr && kv < p.Tk ? ld_nc_i32_here(cols + kv) : -1;
    }
  };
  if constexpr (kQueue) fetch(0);  // on their way while the query token's are (ten registers too many where a warp has few groups: eight caches of 1111 6.2 -> 6.7 us)
  const int qpos = p.q_pos ? min(max(p.q_pos[b], 0), p.Tk - 1) : p.Tk - 1;
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

  // `count` keys of the queue from `first_key` on; slots past the last one repeat it with a score of -inf
  auto take = [&](int first_key, int count) {
    uint4 kr[kUnroll], vr[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int key = s_queue[first_key + min(u * kRows + sub, count - 1)];
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

  // Which keys of the kDecAtOnce groups that `doc` and `col` belong to are allowed, a ballot a group.
  auto allowed = [&](int first, unsigned (&ok)[kDecAtOnce]) {
    unsigned long long word[kDecAtOnce];
#pragma unroll
    for (int u = 0; u < kDecAtOnce; ++u) {
      const int kv = group_at(first, u) * 32 + lane;
      const bool ask = kv <= qpos && doc[u] != qdoc && link_row != nullptr && col[u] >= 0 && col[u] < 64 * p.mask.W;
      word[u] = ask ? static_cast<unsigned long long>(__ldg(link_row + (col[u] >> 6))) : 0ull;
    }
#pragma unroll
    for (int u = 0; u < kDecAtOnce; ++u) {
      const int kv = group_at(first, u) * 32 + lane;
      ok[u] = __ballot_sync(0xffffffffu, kv <= qpos && (doc[u] == qdoc || ((word[u] >> (col[u] & 63)) & 1ull)));
    }
  };
  const unsigned below = (1u << lane) - 1u;
  if constexpr (!kQueue) {
    int* queue = s_queue + warp * (kGroups * 32);
    unsigned ok[kDecAtOnce];
    fetch(0);
    allowed(0, ok);
    int total = 0;
#pragma unroll
    for (int u = 0; u < kDecAtOnce; ++u) {
      if ((ok[u] >> lane) & 1u) queue[total + __popc(ok[u] & below)] = group_at(0, u) * 32 + lane;
      total += __popc(ok[u]);
    }
    __syncwarp();
    int from = 0;
    for (; from + kBatch <= total; from += kBatch) take(warp * (kGroups * 32) + from, kBatch);
    if (from < total) take(warp * (kGroups * 32) + from, total - from);
  } else {
    for (int first = 0; first * cs + blockIdx.x < qpos / 32 + 1; first += kDecWarps * kGroups) {
      if (first > 0) __syncthreads();  // the queue of the last round has been read
      unsigned ok[kGroups / kDecAtOnce][kDecAtOnce];
#pragma unroll
      for (int v = 0; v < kGroups / kDecAtOnce; ++v) {
        const int from = first + v * kDecAtOnce * kDecWarps;
        if (from > 0) fetch(from);
        allowed(from, ok[v]);
#pragma unroll
        for (int u = 0; u < kDecAtOnce; ++u)
          if (lane == 0) s_count[(v * kDecAtOnce + u) * kDecWarps + warp] = __popc(ok[v][u]);
      }
      __syncthreads();
      // Places in the queue by group: a lane adds up four neighbouring counts; this warp's are the same one of each lane's.
      static_assert(kDecWarps % 4 == 0 && kDecWarps * kDecGroups == 128, "");
      const int4 c = reinterpret_cast<const int4*>(s_count)[lane];
      const int four = c.x + c.y + c.z + c.w, mine = warp & 3;
      int upto = four;
#pragma unroll
      for (int x = 1; x < 32; x <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, upto, x);
        if (lane >= x) upto += o;
      }
      const int total = __shfl_sync(0xffffffffu, upto, 31);
      const int before = upto - four + (mine > 0 ? c.x : 0) + (mine > 1 ? c.y : 0) + (mine > 2 ? c.z : 0);
#pragma unroll
      for (int u = 0; u < kGroups; ++u) {
        const unsigned keys = ok[u / kDecAtOnce][u % kDecAtOnce];
        const int place = __shfl_sync(0xffffffffu, before, (u * kDecWarps + warp) / 4);
        if ((keys >> lane) & 1u) s_queue[place + __popc(keys & below)] = group_at(first, u) * 32 + lane;
      }
      __syncthreads();
      int from = warp * kBatch;
      for (; from + kBatch <= total; from += kDecWarps * kBatch) take(from, kBatch);
      if (from < total) take(from, total - from);
    }
  }
  bool bad = false;
#pragma unroll
  for (int i = 0; i < 8; ++i) bad = bad || o[i] != o[i];
  if (__syncthreads_or(bad)) {
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
  cluster_wait();
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
    // blocks -> the first one: written there, so that it reads its own shared memory instead of the others' (two round trips less at the end)
    float* part = cluster.map_shared_rank(&s_part[blockIdx.x][0], 0);
    if (d == 0) { part[0] = mb; part[1] = lb; }
    part[2 + d] = ob;
  }
  cluster_arrive();
  if (blockIdx.x > 0) return;
  cluster_wait();
  if (d < D) {
    float mc = s_part[0][0];
#pragma unroll
    for (int r = 1; r < kDecCluster; ++r) mc = r < cs ? fmaxf(mc, s_part[r][0]) : mc;
    float lc = 0.f, oc = 0.f;
#pragma unroll
    for (int r = 0; r < kDecCluster; ++r) {
      if (r >= cs) break;
      const float mr = s_part[r][0];
      const float f = mr == -CUDART_INF_F ? 0.f : fast_exp2(mr - mc);
      lc = fmaf(f, s_part[r][1], lc);
      oc = fmaf(f, f == 0.f ? 0.f : s_part[r][2 + d], oc);
    }
    p.out[(size_t)b * p.o_sb + (size_t)h * p.o_sh + d] = __float2bfloat16(lc > 0.f ? oc / lc : 0.f);
    if (d == 0) p.lse[(size_t)b * p.H + h] = lc > 0.f ? (mc + log2f(lc)) * 0.6931471805599453f : -CUDART_INF_F;
  }
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
  // Blocks per (batch, head): twice the SM count in all, as long as every warp gets two groups of keys.
  const long long groups = (Tk + 31) / 32;
  int cs = 1;
  while (cs < kDecCluster && (long long)B * H * cs < 2 * 148 && groups >= 2ll * kDecWarps * 2 * cs) cs *= 2;
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
  const bool queue = groups > (long long)cs * kDecWarps * kDecAtOnce;
  // One block an SM where all blocks find a place that way: a cluster needs its SMs in one part of the chip, so 148 single blocks do, 128 in clusters of two or four, 96 of eight, but
  // not 128 of eight.  us, two -> one: all keys of 16 x 1846, H = 8, D = 128 27.0 -> 24.8, 8 x 2000, H = 12 25.7 -> 22.9, 2 x 7723, H = 8 (four) 23.7 -> 21.5, linked 39109, H = 12,
  // D = 64 (eight) 15.9 -> 14.8; beyond the lines all keys of 16 x 2000, H = 12, D = 128 35.8 -> 45.9, 32768, H = 16 (eight) 59.6 -> 83.3.
  const bool alone = (long long)B * H * cs <= (cs == 1 ? 148 : cs < 8 ? 128 : 96);
  using Kernel = void (*)(DecodeParams);
  constexpr Kernel kernels[2][2][2] = {{{decode_kernel<64, false, 2>, decode_kernel<64, false, 1>}, {decode_kernel<64, true, 2>, decode_kernel<64, true, 1>}},
                                       {{decode_kernel<128, false, 2>, decode_kernel<128, false, 1>}, {decode_kernel<128, true, 2>, decode_kernel<128, true, 1>}}};
  if (D != 64 && D != 128) return -142;
  return cudaLaunchKernelEx(&cfg, kernels[D == 128][queue][alone], p) == cudaSuccess ? 0 : -141;
}

}  // namespace ts2ts
