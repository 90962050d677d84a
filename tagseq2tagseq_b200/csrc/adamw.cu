// AdamW over the fp32 parameters of the training step (the reference's parameter groups: main.py:301-337).
//
// In a file of its own because it is compiled without --use_fast_math: root and quotient are rounded correctly and
// subnormal moments stay, as in the optimizer it stands for.  The pass is bound by memory either way.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "launch.cuh"

namespace ts2ts {
namespace {

// One decoupled-weight-decay Adam step over many tensors per launch.  HBM-bound: 28 bytes per parameter.  A block owns
// kAdamChunk consecutive elements of one tensor, two 16-byte vectors of each of the four arrays per thread, all in flight at once.
// us, four such steps a block one after the other -> one: 115 M elements 486 -> 470 (492 at the copy rate), 33.6 M 150 -> 144, 12.6 M 62.5 -> 58.4, 4.2 M 27.6 -> 25.6,
// with one vector a thread (1024 elements a block) 480, 148, 60.4 and 25.6.
constexpr int kAdamTensors = 64, kAdamThreads = 256, kAdamChunk = 8 * kAdamThreads;
struct AdamTensor {
  float* p;
  const float* g;
  float *m, *v;
  int64_t n;
  int first_block;
  float step_size, inv_sqrt_bc2;  // lr / (1 - beta1^t), 1 / sqrt(1 - beta2^t)
};
struct AdamArgs {
  AdamTensor t[kAdamTensors];
  int count;
  float decay, beta1, beta2, rest1, rest2, eps;  // decay = 1 - lr * weight_decay, rest = 1 - beta
};
__device__ __forceinline__ void adam_one(float& p, float g, float& m, float& v, const AdamArgs& a, const AdamTensor& t) {
  p *= a.decay;
  m = a.beta1 * m + a.rest1 * g;
  v = a.beta2 * v + a.rest2 * g * g;
  p -= t.step_size * m / (sqrtf(v) * t.inv_sqrt_bc2 + a.eps);
}
__global__ void __launch_bounds__(kAdamThreads) adamw_kernel(const __grid_constant__ AdamArgs a) {
  wait_previous();
  int lo = 0, hi = a.count - 1;  // last tensor whose first block is not after this one
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (a.t[mid].first_block <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const AdamTensor& t = a.t[lo];
  const int64_t begin = (int64_t)((int)blockIdx.x - t.first_block) * kAdamChunk;
  const int64_t end = min(begin + (int64_t)kAdamChunk, t.n);
  const bool vec = ((reinterpret_cast<uintptr_t>(t.p) | reinterpret_cast<uintptr_t>(t.g) | reinterpret_cast<uintptr_t>(t.m) |
                     reinterpret_cast<uintptr_t>(t.v)) & 15u) == 0;
  int64_t i = begin;
  if (vec) {
    const int64_t vend = begin + (end - begin) / 4 * 4;
    const int64_t j = begin + 4 * threadIdx.x, j2 = j + 4 * kAdamThreads;
    if (j < vend) {
      const bool two = j2 < vend;
      float4 p[2], g[2], m[2], v[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int64_t at = k == 0 || !two ? j : j2;
        p[k] = *reinterpret_cast<const float4*>(t.p + at); g[k] = __ldcs(reinterpret_cast<const float4*>(t.g + at));
        m[k] = *reinterpret_cast<const float4*>(t.m + at); v[k] = *reinterpret_cast<const float4*>(t.v + at);
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (k == 1 && !two) break;
        adam_one(p[k].x, g[k].x, m[k].x, v[k].x, a, t);
        adam_one(p[k].y, g[k].y, m[k].y, v[k].y, a, t);
        adam_one(p[k].z, g[k].z, m[k].z, v[k].z, a, t);
        adam_one(p[k].w, g[k].w, m[k].w, v[k].w, a, t);
        const int64_t at = k == 0 ? j : j2;
        *reinterpret_cast<float4*>(t.p + at) = p[k];
        *reinterpret_cast<float4*>(t.m + at) = m[k];
        *reinterpret_cast<float4*>(t.v + at) = v[k];
      }
    }
    i = vend;
  }
  for (i += threadIdx.x; i < end; i += kAdamThreads) {
    float p = t.p[i], m = t.m[i], v = t.v[i];
    adam_one(p, t.g[i], m, v, a, t);
    t.p[i] = p; t.m[i] = m; t.v[i] = v;
  }
}

}  // namespace

cudaError_t launch_adamw(int count, float* const* p, const float* const* g, float* const* m, float* const* v, const int64_t* n,
                         const float* steps, double lr, double beta1, double beta2, double eps, double weight_decay, cudaStream_t stream) {
  AdamArgs a;
  a.decay = (float)(1.0 - lr * weight_decay); a.beta1 = (float)beta1; a.beta2 = (float)beta2; a.eps = (float)eps;
  a.rest1 = (float)(1.0 - beta1); a.rest2 = (float)(1.0 - beta2);
  for (int done = 0; done < count;) {
    int64_t blocks = 0;
    a.count = 0;
    while (done < count && a.count < kAdamTensors) {
      const int64_t need = (n[done] + kAdamChunk - 1) / kAdamChunk;
      if (a.count > 0 && blocks + need > 0x7fffffff) break;
      if (need > 0) {
        AdamTensor& t = a.t[a.count++];
        t.p = p[done]; t.g = g[done]; t.m = m[done]; t.v = v[done]; t.n = n[done];
        t.first_block = (int)blocks;
        t.step_size = (float)(lr / (1.0 - pow(beta1, (double)steps[done])));
        t.inv_sqrt_bc2 = (float)(1.0 / sqrt(1.0 - pow(beta2, (double)steps[done])));
        blocks += need;
      }
      ++done;
    }
    const cudaError_t e = blocks > 0 ? launch_after(adamw_kernel, dim3((unsigned)blocks), kAdamThreads, 0, stream, a) : cudaSuccess;
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

}  // namespace ts2ts
