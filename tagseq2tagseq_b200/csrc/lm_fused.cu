// Memory-bound pieces of the decoder layer around the attention operator, one pass over HBM each: residual add +
// RMSNorm, rotary embedding applied in place to the q and k parts of the packed QKV projection, SwiGLU, and the
// cross-entropy of the output head.  They stand where the reference's training step has its fused modules
// (model/modules/layer.py:20-35: RMSNorm, rotary attention, SwiGLU; model/modules/training_module.py:205: fused
// linear + cross-entropy loss) and only exist so that the training-step benchmark measures the attention kernels and
// the GEMMs rather than chains of element-wise launches.  All arithmetic is fp32; bf16 only in memory.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <algorithm>

#include "launch.cuh"
#include "ptx.cuh"

namespace ts2ts {
namespace {

template <int N> struct IntTag { static constexpr int value = N; };
constexpr int kMaxVec = 4;  // float4 per thread and row in the wide variant: C <= 16 * blockDim.x

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Block-wide reductions; `red` holds 32 floats; every thread receives the result.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  return warp_sum(lane < nw ? red[lane] : 0.f);
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  return warp_max(lane < nw ? red[lane] : -CUDART_INF_F);
}

__device__ __forceinline__ float4 bf16x4_to_float4(uint2 raw) {
  const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
  const float2 a = __bfloat1622float2(lo), b = __bfloat1622float2(hi);
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ uint2 float4_to_bf16x4(float4 v) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
  uint2 r;
  r.x = *reinterpret_cast<const uint32_t*>(&lo);
  r.y = *reinterpret_cast<const uint32_t*>(&hi);
  return r;
}
__device__ __forceinline__ void bf16x8_to_float(uint4 raw, float (&f)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
    f[2 * i] = a.x;
    f[2 * i + 1] = a.y;
  }
}
__device__ __forceinline__ uint4 float_to_bf16x8(const float (&f)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&p);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// ---------------------------------------------------------------------------------------------- residual add + RMSNorm
// x_out = x_in + a (kAdd, or x_in alone), h = x_out * rstd * w with rstd = 1 / sqrt(mean(x_out^2) + eps).  One block per row.
// With 32 registers two blocks of 1024 threads share an SM: with 40, for the loads of x_in and a of all four vectors at once, they do not (2100 x 16384 69 -> 86 us).
template <int NV, bool kAdd>  // float4 per thread and row: 1 when C <= 4 * blockDim.x, else kMaxVec
__global__ void __launch_bounds__(1024, 2) add_rmsnorm_fwd_kernel(const float* __restrict__ x_in, const __nv_bfloat16* __restrict__ a, const float* __restrict__ w,
                                                                  float* x_out, __nv_bfloat16* __restrict__ h, float* __restrict__ rstd, int C, float eps) {
  __shared__ float red[32];
  const size_t base = (size_t)blockIdx.x * C;
  float4 v[NV];
  float ss = 0.f;
  wait_previous();
  x_in = settled(x_in); a = settled(a); w = settled(w);
  auto load = [&](int c) { return *reinterpret_cast<const float4*>(x_in + base + c); };
  if (!kAdd) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (threadIdx.x + i * blockDim.x) * 4;
      if (c < C) v[i] = load(c);
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * blockDim.x) * 4;
    if (c < C) {
      float4 x;
      if (kAdd) {
        x = load(c);
        const float4 f = bf16x4_to_float4(*reinterpret_cast<const uint2*>(a + base + c));
        x.x += f.x; x.y += f.y; x.z += f.z; x.w += f.w;
      } else {
        x = v[i];
      }
      *reinterpret_cast<float4*>(x_out + base + c) = x;
      v[i] = x;
      ss += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
    }
  }
  ss = block_sum(ss, red);
  const float r = rsqrtf(ss / (float)C + eps);
  if (threadIdx.x == 0) rstd[blockIdx.x] = r;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * blockDim.x) * 4;
    if (c < C) {
      const float4 g = *reinterpret_cast<const float4*>(w + c);
      const float4 x = v[i];
      *reinterpret_cast<uint2*>(h + base + c) = float4_to_bf16x4(make_float4(x.x * r * g.x, x.y * r * g.y, x.z * r * g.z, x.w * r * g.w));
    }
  }
}

// Gradient of the pair above.  With xh = x_out * rstd and g = dh * w:
//   d(x_out) = dx_up + rstd * (g - xh * mean(g * xh)),  dw = sum over rows of dh * xh.
// d(x_out) is the gradient of both x_in and a (written in fp32 and, when da is given, in bf16).  Blocks walk the rows
// with a stride, keep their share of dw in registers and write it to row blockIdx.x of dw_part [gridDim.x, C] at the
// end (atomics on the C addresses of one dw vector serialise a thousand blocks); a second kernel adds the rows up.
//
// HBM-bound, 16 bytes per element: the loads of the next row are on their way while this one is reduced and stored (kAhead; four vectors a
// thread and their successors do not fit the registers: 4096 x 8192 142 -> 230 us), and
// the reduction's scratch alternates so that one barrier per row suffices.  us, two rows at once and none ahead -> one and the next: 16384 x 768 50 -> 46,
// 32768 x 2048 202 -> 175 (164 at the copy rate), 8192 x 4096 126 -> 95, 1024 x 256 13.3 -> 11.3, each with the sum of its weight gradients.
template <int NV, bool kAhead>
__global__ void __launch_bounds__(1024) add_rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dh, const float* __restrict__ dx_up,
                                                               const float* __restrict__ x, const float* __restrict__ w,
                                                               const float* __restrict__ rstd, float* __restrict__ dx,
                                                               __nv_bfloat16* __restrict__ da, float* __restrict__ dw_part, int N, int C) {
  __shared__ float red[2][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float4 wv[NV], acc[NV];
  wait_previous();
  dh = settled(dh); dx_up = settled(dx_up); x = settled(x); w = settled(w); rstd = settled(rstd);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * blockDim.x) * 4;
    wv[i] = c < C ? *reinterpret_cast<const float4*>(w + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  struct Row {  // this thread's part of one, dh as it lies in memory
    float4 x[NV], up[NV];
    uint2 dh[NV];
    float rs;
  } in;
  auto load = [&](int row) {
    in.rs = rstd[row];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (threadIdx.x + i * blockDim.x) * 4;
      in.x[i] = in.up[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      in.dh[i] = make_uint2(0u, 0u);
      if (c < C) {
        const size_t at = (size_t)row * C + c;
        in.x[i] = *reinterpret_cast<const float4*>(x + at);
        in.dh[i] = *reinterpret_cast<const uint2*>(dh + at);
        if (dx_up != nullptr) in.up[i] = *reinterpret_cast<const float4*>(dx_up + at);
      }
    }
  };
  int buf = 0;
  if (kAhead && (int)blockIdx.x < N) load(blockIdx.x);
  for (int row = blockIdx.x; row < N; row += gridDim.x, buf ^= 1) {
    if (!kAhead) load(row);
    const float rs = in.rs;
    float4 xh[NV], g[NV], up[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      xh[i] = in.x[i];
      up[i] = in.up[i];
      g[i] = bf16x4_to_float4(in.dh[i]);
    }
    if (kAhead && row + (int)gridDim.x < N) load(row + gridDim.x);
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float4& h = xh[i];
      float4& d = g[i];
      h.x *= rs; h.y *= rs; h.z *= rs; h.w *= rs;
      acc[i].x += d.x * h.x; acc[i].y += d.y * h.y; acc[i].z += d.z * h.z; acc[i].w += d.w * h.w;
      d.x *= wv[i].x; d.y *= wv[i].y; d.z *= wv[i].z; d.w *= wv[i].w;
      dot += d.x * h.x + d.y * h.y + d.z * h.z + d.w * h.w;
    }
    dot = warp_sum(dot);
    if (lane == 0) red[buf][warp] = dot;
    __syncthreads();
    dot = warp_sum(lane < nw ? red[buf][lane] : 0.f) / (float)C;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (threadIdx.x + i * blockDim.x) * 4;
      if (c < C) {
        const size_t at = (size_t)row * C + c;
        const float4 h = xh[i], d = g[i], u = up[i];
        const float4 o = make_float4(rs * (d.x - h.x * dot) + u.x, rs * (d.y - h.y * dot) + u.y, rs * (d.z - h.z * dot) + u.z, rs * (d.w - h.w * dot) + u.w);
        *reinterpret_cast<float4*>(dx + at) = o;
        if (da != nullptr) *reinterpret_cast<uint2*>(da + at) = float4_to_bf16x4(o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * blockDim.x) * 4;
    if (c < C) *reinterpret_cast<float4*>(dw_part + (size_t)blockIdx.x * C + c) = acc[i];
  }
}
// dw[c] = (`add` to what is there) the sum over the rows of dw_part[rows, C].  A block owns 32 columns: eight lanes of a warp read one row's 128
// bytes, so that 128 rows are in flight per block; one thread per column was a serial chain of loads (66 us per call at
// 1480 x 768, more than the kernel whose partial sums it adds).
__global__ void __launch_bounds__(1024) column_sum_kernel(const float* __restrict__ part, float* dw, int rows, int C, bool add) {
  __shared__ float4 red[32][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 7;
  const int c = blockIdx.x * 32 + sub * 4;
  wait_previous();
  part = settled(part);
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c < C) {
#pragma unroll 4
    for (int r = warp * 4 + (lane >> 3); r < rows; r += 128) {
      const float4 v = *reinterpret_cast<const float4*>(part + (size_t)r * C + c);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
  }
#pragma unroll
  for (int o = 8; o < 32; o <<= 1) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
    s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    s.z += __shfl_xor_sync(0xffffffffu, s.z, o);
    s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
  }
  if (lane < 8) red[warp][lane] = s;
  __syncthreads();
  if (threadIdx.x < 32) {  // thread = column
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) t += reinterpret_cast<const float*>(red[i])[threadIdx.x];
    const int col = blockIdx.x * 32 + threadIdx.x;
    if (col < C) dw[col] = add ? dw[col] + t : t;
  }
}

// ---------------------------------------------------------------------------------------------- copies of many tensors
// All of a step's weights to bf16, or all gradients of a step as they are, in one launch instead of one each: a block takes kMoveBytes consecutive bytes of
// one source.  HBM-bound, 6 and 8 bytes an element.  us, bf16: the 17 weights of four layers at d_model 768 with 50304 words (76 M elements, 70 at the copy rate)
// 111 -> 72; nine of 3.6 M in all 17 in nine launches, below 5 in one.  Copies: 15 gradients of 3.6 M elements and the loss 13.6 + 1.4 by torch's launches -> 7.
constexpr int kMoveTensors = 128, kMoveThreads = 256, kMoveBytes = 32768;
struct MoveArgs {
  const void* src[kMoveTensors];
  void* dst[kMoveTensors];
  int64_t n[kMoveTensors];  // elements to convert, or bytes to copy
  int first_block[kMoveTensors];
  int count;
};
__device__ __forceinline__ void move_cast(const float* src, __nv_bfloat16* dst, int64_t begin, int64_t end) {
  int64_t i = begin;
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0) {
    const int64_t vend = begin + (end - begin) / 8 * 8;
#pragma unroll 4
    for (int64_t j = begin + 8 * threadIdx.x; j < vend; j += 8 * kMoveThreads) {
      float f[8];
      *reinterpret_cast<float4*>(f) = *reinterpret_cast<const float4*>(src + j);
      *reinterpret_cast<float4*>(f + 4) = *reinterpret_cast<const float4*>(src + j + 4);
      *reinterpret_cast<uint4*>(dst + j) = float_to_bf16x8(f);
    }
    i = vend;
  }
  for (i += threadIdx.x; i < end; i += kMoveThreads) dst[i] = __float2bfloat16_rn(src[i]);
}
// Bytes from `begin` on in pieces of Unit; returns where the last whole one ends.
template <typename Unit> __device__ __forceinline__ int64_t move_units(const char* src, char* dst, int64_t begin, int64_t end) {
  const int64_t uend = begin + (end - begin) / (int64_t)sizeof(Unit) * (int64_t)sizeof(Unit);
#pragma unroll 8
  for (int64_t j = begin + (int64_t)sizeof(Unit) * threadIdx.x; j < uend; j += sizeof(Unit) * kMoveThreads)
    *reinterpret_cast<Unit*>(dst + j) = *reinterpret_cast<const Unit*>(src + j);
  return uend;
}
template <bool kCast>
__global__ void __launch_bounds__(kMoveThreads) move_kernel(const __grid_constant__ MoveArgs a) {
  int lo = 0, hi = a.count - 1;  // last tensor whose first block is not after this one
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (a.first_block[mid] <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  wait_previous();
  constexpr int kChunk = kCast ? kMoveBytes / 4 : kMoveBytes;
  const void* src = settled(a.src[lo]);
  const int64_t begin = (int64_t)((int)blockIdx.x - a.first_block[lo]) * kChunk, end = min(begin + (int64_t)kChunk, a.n[lo]);
  if constexpr (kCast) {
    move_cast(static_cast<const float*>(src), static_cast<__nv_bfloat16*>(a.dst[lo]), begin, end);
  } else {
    const char* from = static_cast<const char*>(src);
    char* to = static_cast<char*>(a.dst[lo]);
    const uintptr_t at = reinterpret_cast<uintptr_t>(from) | reinterpret_cast<uintptr_t>(to);
    int64_t i = begin;
    if ((at & 15u) == 0) i = move_units<uint4>(from, to, i, end);
    else if ((at & 3u) == 0) i = move_units<uint32_t>(from, to, i, end);
    move_units<char>(from, to, i, end);
  }
}

// ---------------------------------------------------------------------------------------------- rotary embedding
// In place on the q (part 0) and k (part 1) slices of qkv [B,T,3,H,D]: pairs (i, i + D/2),
//   y1 = x1 cos - sign * x2 sin,  y2 = x2 cos + sign * x1 sin;  sign = -1 turns a gradient back (the inverse rotation).
// cos / sin are fp32 [T, D/2].  One thread rotates eight pairs.
__global__ void rope_qk_kernel(__nv_bfloat16* qkv, const float* __restrict__ cs, const float* __restrict__ sn, int T, int H, int D,
                               int64_t n_threads, float sign) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  wait_previous();
  cs = settled(cs); sn = settled(sn);
  if (idx >= n_threads) return;
  const int vec_per_head = D / 16;  // groups of eight pairs
  int64_t r = idx;
  const int i8 = (int)(r % vec_per_head); r /= vec_per_head;
  const int h = (int)(r % H); r /= H;
  const int part = (int)(r % 2); r /= 2;
  const int t = (int)(r % T);
  const int64_t b = r / T;
  __nv_bfloat16* lo = qkv + ((((b * T + t) * 3 + part) * H + h) * (int64_t)D + i8 * 8);
  __nv_bfloat16* hi = lo + D / 2;
  float x1[8], x2[8], c[8], s[8];
  bf16x8_to_float(*reinterpret_cast<const uint4*>(lo), x1);
  bf16x8_to_float(*reinterpret_cast<const uint4*>(hi), x2);
  const float* cp = cs + (size_t)t * (D / 2) + i8 * 8;
  const float* sp = sn + (size_t)t * (D / 2) + i8 * 8;
  *reinterpret_cast<float4*>(c) = *reinterpret_cast<const float4*>(cp);
  *reinterpret_cast<float4*>(c + 4) = *reinterpret_cast<const float4*>(cp + 4);
  *reinterpret_cast<float4*>(s) = *reinterpret_cast<const float4*>(sp);
  *reinterpret_cast<float4*>(s + 4) = *reinterpret_cast<const float4*>(sp + 4);
  float y1[8], y2[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    y1[i] = x1[i] * c[i] - sign * x2[i] * s[i];
    y2[i] = x2[i] * c[i] + sign * x1[i] * s[i];
  }
  *reinterpret_cast<uint4*>(lo) = float_to_bf16x8(y1);
  *reinterpret_cast<uint4*>(hi) = float_to_bf16x8(y2);
}

// ---------------------------------------------------------------------------------------------- SwiGLU
// gu [N, 2F]: gate in the first F columns, up in the last F (torch.chunk(2, dim=-1));  act = silu(gate) * up.
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ act, int F, int64_t n_vec) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  wait_previous();
  gu = settled(gu);
  if (idx >= n_vec) return;
  const int per_row = F / 8;
  const int64_t row = idx / per_row;
  const int c = (int)(idx % per_row) * 8;
  float g[8], u[8], o[8];
  bf16x8_to_float(*reinterpret_cast<const uint4*>(gu + row * 2 * F + c), g);
  bf16x8_to_float(*reinterpret_cast<const uint4*>(gu + row * 2 * F + F + c), u);
#pragma unroll
  for (int i = 0; i < 8; ++i) o[i] = g[i] / (1.f + __expf(-g[i])) * u[i];
  *reinterpret_cast<uint4*>(act + row * F + c) = float_to_bf16x8(o);
}
// d gate = dact * up * s * (1 + gate * (1 - s)),  d up = dact * gate * s,  s = sigmoid(gate).
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ dact,
                                  __nv_bfloat16* __restrict__ dgu, int F, int64_t n_vec) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  wait_previous();
  gu = settled(gu); dact = settled(dact);
  if (idx >= n_vec) return;
  const int per_row = F / 8;
  const int64_t row = idx / per_row;
  const int c = (int)(idx % per_row) * 8;
  float g[8], u[8], d[8], dg[8], du[8];
  bf16x8_to_float(*reinterpret_cast<const uint4*>(gu + row * 2 * F + c), g);
  bf16x8_to_float(*reinterpret_cast<const uint4*>(gu + row * 2 * F + F + c), u);
  bf16x8_to_float(*reinterpret_cast<const uint4*>(dact + row * F + c), d);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float s = 1.f / (1.f + __expf(-g[i]));
    dg[i] = d[i] * u[i] * s * (1.f + g[i] * (1.f - s));
    du[i] = d[i] * g[i] * s;
  }
  *reinterpret_cast<uint4*>(dgu + row * 2 * F + c) = float_to_bf16x8(dg);
  *reinterpret_cast<uint4*>(dgu + row * 2 * F + F + c) = float_to_bf16x8(du);
}

// ---------------------------------------------------------------------------------------------- cross-entropy
// One block per row of logits [N, V] (bf16, V a multiple of 8).  Forward: lse = log sum exp, loss = lse - logit[target].
__global__ void ce_fwd_kernel(const __nv_bfloat16* __restrict__ logits, const int64_t* __restrict__ target, float* __restrict__ lse,
                              float* __restrict__ loss, int V) {
  __shared__ float red[32];
  wait_previous();
  logits = settled(logits); target = settled(target);
  const __nv_bfloat16* row = logits + (size_t)blockIdx.x * V;
  float m = -CUDART_INF_F, s = 0.f;
  for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) {
    float f[8];
    bf16x8_to_float(*reinterpret_cast<const uint4*>(row + c), f);
    float mx = f[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) mx = fmaxf(mx, f[i]);
    const float m_new = fmaxf(m, mx);
    if (m_new == -CUDART_INF_F) continue;  // nothing but -inf so far: contributes nothing, and -inf - -inf is no number
    float add = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) add += __expf(f[i] - m_new);
    s = s * __expf(m - m_new) + add;
    m = m_new;
  }
  const float m_all = block_max(m, red);
  const float s_all = block_sum(m == -CUDART_INF_F ? 0.f : s * __expf(m - m_all), red);
  if (threadIdx.x == 0) {
    const float l = m_all + logf(s_all);
    const int64_t tg = target[blockIdx.x];
    lse[blockIdx.x] = l;
    loss[blockIdx.x] = (tg >= 0 && tg < V) ? l - __bfloat162float(row[tg]) : 0.f;
  }
}
// Backward, in place: logits <- (softmax - onehot(target)) * gscale[0] * inv_n.  Rows whose target is out of range
// contributed no loss and get a zero gradient.
__global__ void ce_bwd_kernel(__nv_bfloat16* logits, const int64_t* __restrict__ target, const float* __restrict__ lse,
                              const float* __restrict__ gscale, float inv_n, int V) {
  wait_previous();
  target = settled(target); lse = settled(lse); gscale = settled(gscale);
  __nv_bfloat16* row = logits + (size_t)blockIdx.x * V;
  const int64_t tg = target[blockIdx.x];
  const bool live = tg >= 0 && tg < V;
  const float l = lse[blockIdx.x], g = live ? gscale[0] * inv_n : 0.f;
  for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) {
    float f[8];
    bf16x8_to_float(*reinterpret_cast<const uint4*>(row + c), f);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = (__expf(f[i] - l) - ((int64_t)(c + i) == tg ? 1.f : 0.f)) * g;
    *reinterpret_cast<uint4*>(row + c) = float_to_bf16x8(f);
  }
}

// Loss and gradient of a row in one pass: the row (at most kCeRowBytes) is brought into shared memory once, read there
// for the log-sum-exp and again for the gradient, which is written over the logits.  HBM-bound, 4 bytes per logit
// instead of the 6 of the two kernels above; two blocks of a 50304-logit row share an SM, so that one's copy overlaps the
// other's arithmetic.  The gradient is that of the mean loss (times inv_n, not times what reaches the loss from above).
// What is left beside the copy are two exponentials a logit: maxima are taken of bf16 pairs, four vectors of a thread between two looks at the
// running one, difference and scale are packed, only the target's vector knows of it.  A row of up to 1024 vectors of eight has 64 threads (up to 16 vectors each), up to 2048
// 128, up to 4096 256 (8 to 16 each), beyond 512 (8 to 27).
// us (floor at the copy rate; one comparison and a maximum a logit, 512 threads whatever the row -> now): 16384 x 50304 (504) 650 -> 557, x 32768 (328) 422 -> 338,
// x 16384 (164) 235 -> 167, x 4096 (41) 120 -> 50; 1024 x 4096 (3) 15.8 -> 12.8.  512 threads for x 32768 343, 256 for x 50304 574.
constexpr int kCeRowBytes = 216 * 1024;
constexpr uint32_t kNoLogits = 0xff80ff80u;  // two of -inf
constexpr float kLog2e = 1.4426950408889634f;
template <int kN>
__device__ __forceinline__ float max_bf16x8(const uint4 (&raw)[kN]) {
  __nv_bfloat162 most = *reinterpret_cast<const __nv_bfloat162*>(&raw[0].x);
#pragma unroll
  for (int u = 0; u < kN; ++u) {
    const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) most = __hmax2(most, *reinterpret_cast<const __nv_bfloat162*>(&w[i]));
  }
  return fmaxf(__low2float(most), __high2float(most));
}
// exp(f - most) of eight values, two to an operation.  The difference is taken before the scaling: where logits are large (the lowest value stands for a class that is
// ruled out) a scaled maximum is off by more than an exponent can be, or past what fp32 holds.  One multiply-add for both would save 1 % (16384 x 50304 552 us).
__device__ __forceinline__ void exp_bf16x8(uint4 raw, float most, float (&e)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  const unsigned long long scale2 = pack_f32x2(kLog2e, kLog2e), less2 = pack_f32x2(-most, -most);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a, b;
    unpack_f32x2(mul_f32x2(add_f32x2(pack_f32x2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u)), less2), scale2), a, b);
    e[2 * i] = fast_exp2(a);
    e[2 * i + 1] = fast_exp2(b);
  }
}
template <int kThreads, int kChunks>
__global__ void __launch_bounds__(kThreads) ce_fwd_grad_kernel(__nv_bfloat16* logits, const int64_t* __restrict__ target,
                                                                 float* __restrict__ loss, float inv_n, int V) {
  extern __shared__ __align__(128) uint8_t ce_row[];
  __shared__ __align__(8) uint64_t bars[kChunks];
  __shared__ float red_m[kThreads / 32], red_s[kThreads / 32];
  __shared__ int late;
  __nv_bfloat16* row = logits + (size_t)blockIdx.x * V;
  const int n_vec = V / 8, per_chunk = (n_vec + kChunks - 1) / kChunks;  // in 16-byte vectors
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  wait_previous();
  target = settled(target);
  if (tid == 0) {
    late = 0;
    for (int k = 0; k < kChunks; ++k) mbar_init(&bars[k], 1);
    fence_mbar_init();
    for (int k = 0; k < kChunks; ++k) {
      const int first = min(k * per_chunk, n_vec), count = min(per_chunk, n_vec - first);
      mbar_expect_tx(&bars[k], count * 16);
      if (count > 0) bulk_load(ce_row + first * 16, row + first * 8, count * 16, &bars[k]);
    }
  }
  const int64_t tg = target[blockIdx.x];
  const bool live = tg >= 0 && tg < V;
  __syncthreads();
  const uint4* sv = reinterpret_cast<const uint4*>(ce_row);
  float m = -CUDART_INF_F, s = 0.f;
  // up to kN vectors of this thread's, `kThreads` apart
  auto sum_up = [&](auto vecs, int c, int end) {
    constexpr int kN = decltype(vecs)::value;
    uint4 raw[kN];
#pragma unroll
    for (int u = 0; u < kN; ++u) raw[u] = u == 0 || c + u * kThreads < end ? sv[c + u * kThreads] : make_uint4(kNoLogits, kNoLogits, kNoLogits, kNoLogits);
    const float m_new = fmaxf(m, max_bf16x8(raw));
    if (m_new == -CUDART_INF_F) return;
    unsigned long long sum[2] = {0ull, 0ull};
#pragma unroll
    for (int u = 0; u < kN; ++u) {
      float e[8];
      exp_bf16x8(raw[u], m_new, e);
#pragma unroll
      for (int i = 0; i < 8; i += 2) sum[(i >> 1) & 1] = add_f32x2(sum[(i >> 1) & 1], pack_f32x2(e[i], e[i + 1]));
    }
    float a, b;
    unpack_f32x2(add_f32x2(sum[0], sum[1]), a, b);
    s = s * __expf(m - m_new) + (a + b);
    m = m_new;
  };
  bool ok = true;
  for (int k = 0; k < kChunks; ++k) {
    ok = ok && mbar_wait(&bars[k], 0, &late, 1);
    if (!ok) break;
    const int end = min((k + 1) * per_chunk, n_vec);
    int c = k * per_chunk + tid;
    for (; c + 2 * kThreads < end; c += 4 * kThreads) sum_up(IntTag<4>{}, c, end);
    if (c + kThreads < end) sum_up(IntTag<2>{}, c, end);
    else if (c < end) sum_up(IntTag<1>{}, c, end);
  }
  const float wm = warp_max(m);
  s = warp_sum(m == -CUDART_INF_F ? 0.f : s * __expf(m - wm));
  if (lane == 0) { red_m[warp] = wm; red_s[warp] = s; }
  __syncthreads();
  const float pm = lane < kThreads / 32 ? red_m[lane] : -CUDART_INF_F;
  const float m_all = warp_max(pm);
  const float s_all = warp_sum(pm == -CUDART_INF_F ? 0.f : red_s[lane] * __expf(pm - m_all));
  const float l = m_all + logf(s_all);
  const float hit = live ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(ce_row)[tg]) : 0.f;
  if (tid == 0) loss[blockIdx.x] = !ok ? CUDART_NAN_F : live ? l - hit : 0.f;  // a copy that never came shows as a loss that is no number
  if (!ok) {  // let the copy land before the block's shared memory is released
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    return;
  }
  const float g = live ? inv_n : 0.f;
  const unsigned long long scale2 = pack_f32x2(g, g);
  const int hit_vec = live ? static_cast<int>(tg >> 3) : -1;
#pragma unroll 2
  for (int c = tid; c < n_vec; c += kThreads) {
    float f[8];
    exp_bf16x8(sv[c], l, f);
    if (c != hit_vec) {
#pragma unroll
      for (int i = 0; i < 8; i += 2) unpack_f32x2(mul_f32x2(pack_f32x2(f[i], f[i + 1]), scale2), f[i], f[i + 1]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = (f[i] - (i == static_cast<int>(tg & 7) ? 1.f : 0.f)) * g;
    }
    reinterpret_cast<uint4*>(row)[c] = float_to_bf16x8(f);
  }
}

// x *= gscale[0], and out = bf16(x * gscale[0]).  The first does nothing when the factor is one, which it is unless the
// caller scaled the loss.
__global__ void __launch_bounds__(256) scale_f32_kernel(float* x, const float* __restrict__ gscale, int64_t n) {
  wait_previous();
  gscale = settled(gscale);
  const float g = gscale[0];
  if (g == 1.f) return;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) x[i] *= g;
}
__global__ void __launch_bounds__(256) scale_to_bf16_kernel(const float* __restrict__ x, const float* __restrict__ gscale,
                                                            __nv_bfloat16* __restrict__ out, int64_t n_vec) {
  wait_previous();
  x = settled(x); gscale = settled(gscale);
  const float g = gscale[0];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_vec) return;
  float f[8];
  *reinterpret_cast<float4*>(f) = reinterpret_cast<const float4*>(x)[2 * i];
  *reinterpret_cast<float4*>(f + 4) = reinterpret_cast<const float4*>(x)[2 * i + 1];
#pragma unroll
  for (int k = 0; k < 8; ++k) f[k] *= g;
  reinterpret_cast<uint4*>(out)[i] = float_to_bf16x8(f);
}

// ---------------------------------------------------------------------------------------------- embedding
// dw[v] = the sum of dx[n] over the tokens n with idx[n] == v, added up in an order that depends on idx alone, so that a
// step repeats bit for bit (atomic additions in the order of arrival do not).  Block (bucket, columns) owns 512 columns of
// the ids v with v % kEmbBuckets == bucket: it reads all of idx, 8 bytes a token from L2, and queues its tokens in
// ascending order; a warp then adds up one id's rows at a time.  Ids of more than kEmbHeavy queued rows are shared by the
// block: each warp takes a stretch of the queue, and the sixteen partial rows are added in order.  dw is zeroed before.
// HBM-bound (dx read once, dw written twice at most).  Pass with its memset, uniform ids into 50304 rows: 69 us at
// 16384 x 768, 208 us at 32768 x 2048 (atomics in the order of arrival 51 and 181 us; torch's kernel, which sorts the
// tokens, 371 and 1317 us).  One id for all tokens is the worst case, 700 us at 16384 x 768.
constexpr int kEmbBuckets = 256, kEmbThreads = 512, kEmbWarps = kEmbThreads / 32, kEmbEach = 4, kEmbStep = kEmbEach * kEmbThreads;
constexpr int kEmbList = kEmbStep + 1024, kEmbVec = 4, kEmbCols = 128 * kEmbVec, kEmbHeavy = 64;
__device__ __forceinline__ void add4(float4& a, const float4& b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
__global__ void __launch_bounds__(kEmbThreads) embedding_bwd_kernel(const int64_t* __restrict__ idx, const float* __restrict__ dx, float* dw, int N,
                                                                    int C, int64_t V) {
  __shared__ int s_pos[kEmbList], s_id[kEmbList], s_cnt[2][kEmbEach * kEmbWarps], s_n[2];
  __shared__ unsigned short s_lead[kEmbList], s_heavy[kEmbList / kEmbHeavy];
  __shared__ float4 s_part[kEmbWarps][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, bucket = blockIdx.x;
  const int col = blockIdx.y * kEmbCols + lane * 4;  // of this lane's first vector; the others follow 128 columns apart
  int count = 0;                                     // queued tokens, the same in every thread
  bool first = true;                                 // nothing of this block's rows written yet
  wait_previous();
  idx = settled(idx);  // where dx is read depends on it; dx settled, too, cost registers (spills: 32768 x 2048 207 -> 231 us)

  // sum of the queued rows of `id` between two places of the queue, `kVecs` vectors a lane from vector `from` on
  auto sum_rows = [&](auto vecs, int id, int begin, int end, int from, float4* acc) {
    constexpr int kVecs = decltype(vecs)::value, kAhead = 8 / kVecs;
    for (int at = begin; at < end; at += 32) {
      unsigned hits = __ballot_sync(0xffffffffu, at + lane < end && s_id[at + lane] == id);
      while (hits) {
        float4 row[kAhead][kVecs];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
          const int64_t n = hits ? s_pos[at + __ffs(hits) - 1] : -1;
          hits &= hits - 1;
#pragma unroll
          for (int j = 0; j < kVecs; ++j) {
            const int c = col + 128 * (from + j);
            row[k][j] = n >= 0 && c < C ? __ldg(reinterpret_cast<const float4*>(dx + n * C + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
#pragma unroll
          for (int j = 0; j < kVecs; ++j) add4(acc[j], row[k][j]);
      }
    }
  };
  auto put = [&](int id, int j, float4 v) {
    const int c = col + 128 * j;
    if (c >= C) return;
    float4* out = reinterpret_cast<float4*>(dw + (int64_t)id * C + c);
    if (!first) add4(v, *out);
    *out = v;
  };
  // every id of the queue, whose places are complete and visible
  auto flush = [&]() {
    if (tid < 2) s_n[tid] = 0;
    __syncthreads();
    for (int e = tid; e < count; e += kEmbThreads) {
      const int id = s_id[e];
      int k = 0;
      while (s_id[k] != id) ++k;
      if (k == e) s_lead[atomicAdd(&s_n[0], 1)] = static_cast<unsigned short>(e);
    }
    __syncthreads();
    const int leads = s_n[0];
    for (int u = warp; u < leads; u += kEmbWarps) {
      const int e = s_lead[u], id = s_id[e];
      int rows = 0;
      for (int at = e; at < count; at += 32) rows += __popc(__ballot_sync(0xffffffffu, at + lane < count && s_id[at + lane] == id));
      if (rows > kEmbHeavy) {
        if (lane == 0) s_heavy[atomicAdd(&s_n[1], 1)] = static_cast<unsigned short>(e);
        continue;
      }
      float4 acc[kEmbVec];
#pragma unroll
      for (int j = 0; j < kEmbVec; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      sum_rows(IntTag<kEmbVec>{}, id, e, count, 0, acc);
#pragma unroll
      for (int j = 0; j < kEmbVec; ++j) put(id, j, acc[j]);
    }
    __syncthreads();
    const int heavy = s_n[1], share = (count + kEmbWarps - 1) / kEmbWarps;
    for (int u = 0; u < heavy * kEmbVec; ++u) {
      const int id = s_id[s_heavy[u / kEmbVec]], j = u % kEmbVec;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      sum_rows(IntTag<1>{}, id, warp * share, min((warp + 1) * share, count), j, &acc);
      s_part[warp][lane] = acc;
      __syncthreads();
      if (warp == 0) {
        for (int w = 1; w < kEmbWarps; ++w) add4(acc, s_part[w][lane]);
        put(id, j, acc);
      }
      __syncthreads();
    }
    first = false;
    count = 0;
  };

  int64_t next[kEmbEach];
  auto fetch = [&](int base) {
#pragma unroll
    for (int k = 0; k < kEmbEach; ++k) {
      const int64_t n = (int64_t)base + k * kEmbThreads + tid;
      next[k] = n < N ? __ldg(idx + n) : -1;
    }
  };
  fetch(0);
  int buf = 0;
  for (int64_t base = 0; base < N; base += kEmbStep, buf ^= 1) {
    int64_t v[kEmbEach];
    unsigned mine[kEmbEach];
#pragma unroll
    for (int k = 0; k < kEmbEach; ++k) {
      v[k] = next[k];
      mine[k] = __ballot_sync(0xffffffffu, v[k] >= 0 && v[k] < V && (v[k] & (kEmbBuckets - 1)) == bucket);
      if (lane == 0) s_cnt[buf][k * kEmbWarps + warp] = __popc(mine[k]);
    }
    if (base + kEmbStep < N) fetch((int)(base + kEmbStep));
    __syncthreads();
    // places in the queue: by stretch of 512 tokens, then by warp, then by lane
    const int lo = s_cnt[buf][2 * lane], both = lo + s_cnt[buf][2 * lane + 1];
    int upto = both;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, upto, s);
      if (lane >= s) upto += o;
    }
#pragma unroll
    for (int k = 0; k < kEmbEach; ++k) {
      const int slot = k * kEmbWarps + warp;
      int at = __shfl_sync(0xffffffffu, upto - both, slot / 2) + (slot & 1 ? __shfl_sync(0xffffffffu, lo, slot / 2) : 0);
      if ((mine[k] >> lane) & 1u) {
        at += count + __popc(mine[k] & ((1u << lane) - 1u));
        s_pos[at] = (int)(base + k * kEmbThreads + tid);
        s_id[at] = (int)v[k];
      }
    }
    count += __shfl_sync(0xffffffffu, upto, 31);
    if (count > kEmbList - kEmbStep) {
      __syncthreads();
      flush();
      __syncthreads();
    }
  }
  if (count > 0) {
    __syncthreads();
    flush();
  }
}

int norm_threads(int C) {
  int t = (C / 4 + kMaxVec - 1) / kMaxVec;  // threads needed with kMaxVec float4 each
  t = ((t + 31) / 32) * 32;
  // prefer one float4 per thread while the block stays within 1024 threads
  const int one = ((C / 4 + 31) / 32) * 32;
  return one <= 1024 ? one : t;
}

}  // namespace

cudaError_t launch_add_rmsnorm_fwd(const float* x_in, const void* a, const float* w, float* x_out, void* h, float* rstd, int N, int C,
                                   float eps, cudaStream_t stream) {
  const int threads = norm_threads(C);
  const auto kernel = C <= 4 * threads ? a != nullptr ? add_rmsnorm_fwd_kernel<1, true> : add_rmsnorm_fwd_kernel<1, false>
                                       : a != nullptr ? add_rmsnorm_fwd_kernel<kMaxVec, true> : add_rmsnorm_fwd_kernel<kMaxVec, false>;
  return launch_after(kernel, dim3(N), threads, 0, stream, x_in, static_cast<const __nv_bfloat16*>(a), w, x_out, static_cast<__nv_bfloat16*>(h), rstd, C, eps);
}

// Blocks of the backward kernel = rows of its dw_part workspace.
int add_rmsnorm_bwd_blocks(int64_t N, int C) {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    sms = n;
  }
  const int threads = norm_threads(C);
  const int per_sm = threads >= 1024 ? 1 : 1024 / threads;  // resident blocks at up to 64 registers a thread
  const int64_t cap = (int64_t)sms * per_sm;
  int64_t want = (N + 3) / 4;  // four rows a block or more, once every SM has two: its partial dw row costs traffic of its own
  if (want < 2 * sms) want = N < 2 * sms ? N : 2 * sms;
  return (int)(want < cap ? want : cap);
}

cudaError_t launch_add_rmsnorm_bwd(const void* dh, const float* dx_up, const float* x, const float* w, const float* rstd, float* dx,
                                   void* da, float* dw, bool add, float* dw_part, int N, int C, cudaStream_t stream) {
  const int grid = add_rmsnorm_bwd_blocks(N, C);
  const int threads = norm_threads(C);
  const __nv_bfloat16* g = static_cast<const __nv_bfloat16*>(dh);
  __nv_bfloat16* a = static_cast<__nv_bfloat16*>(da);
  const cudaError_t e = launch_after(C <= 4 * threads ? add_rmsnorm_bwd_kernel<1, true> : add_rmsnorm_bwd_kernel<kMaxVec, false>, dim3(grid), threads, 0, stream,
                                     g, dx_up, x, w, rstd, dx, a, dw_part, N, C);
  return e != cudaSuccess ? e : launch_after(column_sum_kernel, dim3((C + 31) / 32), 1024, 0, stream, dw_part, dw, grid, C, add);
}

template <bool kCast>
cudaError_t launch_move(int count, const void* const* src, void* const* dst, const int64_t* n, cudaStream_t stream) {
  constexpr int kChunk = kCast ? kMoveBytes / 4 : kMoveBytes;
  MoveArgs a;
  for (int done = 0; done < count;) {
    int64_t blocks = 0;
    a.count = 0;
    for (; done < count && a.count < kMoveTensors; ++done) {
      const int64_t need = (n[done] + kChunk - 1) / kChunk;
      if (need == 0) continue;
      if (a.count > 0 && blocks + need > 0x7fffffff) break;
      a.src[a.count] = src[done]; a.dst[a.count] = dst[done]; a.n[a.count] = n[done];
      a.first_block[a.count++] = (int)blocks;
      blocks += need;
    }
    const cudaError_t e = blocks > 0 ? launch_after(move_kernel<kCast>, dim3((unsigned)blocks), kMoveThreads, 0, stream, a) : cudaSuccess;
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
cudaError_t launch_cast_bf16(int count, const float* const* src, void* const* dst, const int64_t* n, cudaStream_t stream) {
  return launch_move<true>(count, reinterpret_cast<const void* const*>(src), dst, n, stream);
}
cudaError_t launch_copy(int count, const void* const* src, void* const* dst, const int64_t* bytes, cudaStream_t stream) {
  return launch_move<false>(count, src, dst, bytes, stream);
}

cudaError_t launch_rope_qk(void* qkv, const float* cs, const float* sn, int B, int T, int H, int D, float sign, cudaStream_t stream) {
  const int64_t n = (int64_t)B * T * 2 * H * (D / 16);
  const int threads = 256;
  return launch_after(rope_qk_kernel, dim3((unsigned)((n + threads - 1) / threads)), threads, 0, stream, static_cast<__nv_bfloat16*>(qkv), cs, sn, T, H, D, n, sign);
}

cudaError_t launch_swiglu_fwd(const void* gu, void* act, int64_t N, int F, cudaStream_t stream) {
  const int64_t n = N * (F / 8);
  const int threads = 256;
  return launch_after(swiglu_fwd_kernel, dim3((unsigned)((n + threads - 1) / threads)), threads, 0, stream, static_cast<const __nv_bfloat16*>(gu),
                      static_cast<__nv_bfloat16*>(act), F, n);
}

cudaError_t launch_swiglu_bwd(const void* gu, const void* dact, void* dgu, int64_t N, int F, cudaStream_t stream) {
  const int64_t n = N * (F / 8);
  const int threads = 256;
  return launch_after(swiglu_bwd_kernel, dim3((unsigned)((n + threads - 1) / threads)), threads, 0, stream, static_cast<const __nv_bfloat16*>(gu),
                      static_cast<const __nv_bfloat16*>(dact), static_cast<__nv_bfloat16*>(dgu), F, n);
}

cudaError_t launch_ce_fwd(const void* logits, const int64_t* target, float* lse, float* loss, int N, int V, cudaStream_t stream) {
  return launch_after(ce_fwd_kernel, dim3(N), 256, 0, stream, static_cast<const __nv_bfloat16*>(logits), target, lse, loss, V);
}

cudaError_t launch_ce_bwd(void* logits, const int64_t* target, const float* lse, const float* gscale, float inv_n, int N, int V,
                          cudaStream_t stream) {
  return launch_after(ce_bwd_kernel, dim3(N), 256, 0, stream, static_cast<__nv_bfloat16*>(logits), target, lse, gscale, inv_n, V);
}

// -1000: the row does not fit shared memory (the caller takes the two-kernel path).
int launch_ce_fwd_grad(void* logits, const int64_t* target, float* loss, float inv_n, int N, int V, cudaStream_t stream) {
  const int bytes = 2 * V;
  if (bytes > kCeRowBytes) return -1000;
  using Kernel = void (*)(__nv_bfloat16*, const int64_t*, float*, float, int);
  constexpr Kernel kernels[5] = {ce_fwd_grad_kernel<64, 1>, ce_fwd_grad_kernel<64, 4>, ce_fwd_grad_kernel<128, 4>, ce_fwd_grad_kernel<256, 4>, ce_fwd_grad_kernel<512, 4>};
  const int n_vec = V / 8, which = n_vec <= 256 ? 0 : n_vec <= 1024 ? 1 : n_vec <= 2048 ? 2 : n_vec <= 4096 ? 3 : 4;
  static bool attr_done[64][5] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return -50;
  if (!attr_done[dev][which]) {
    if (cudaFuncSetAttribute(kernels[which], cudaFuncAttributeMaxDynamicSharedMemorySize, kCeRowBytes) != cudaSuccess) return -50;
    attr_done[dev][which] = true;
  }
  return launch_after(kernels[which], dim3(N), which == 0 ? 64 : 32 << which, bytes, stream, static_cast<__nv_bfloat16*>(logits), target, loss, inv_n, V) == cudaSuccess ? 0 : -50;
}

cudaError_t launch_scale(float* x, void* out_bf16, const float* gscale, int64_t n, cudaStream_t stream) {
  if (out_bf16 == nullptr) {
    const int64_t blocks = (n + 1023) / 1024;
    return launch_after(scale_f32_kernel, dim3((unsigned)(blocks < 1184 ? blocks : 1184)), 256, 0, stream, x, gscale, n);
  }
  return launch_after(scale_to_bf16_kernel, dim3((unsigned)((n / 8 + 255) / 256)), 256, 0, stream, x, gscale, static_cast<__nv_bfloat16*>(out_bf16), n / 8);
}

cudaError_t launch_embedding_bwd(const int64_t* idx, const float* dx, float* dw, int64_t N, int C, int64_t V, cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(dw, 0, (size_t)V * C * sizeof(float), stream);
  if (e != cudaSuccess) return e;
  return launch_after(embedding_bwd_kernel, dim3(kEmbBuckets, (C + kEmbCols - 1) / kEmbCols), kEmbThreads, 0, stream, idx, dx, dw, (int)N, C, V);
}

}  // namespace ts2ts
