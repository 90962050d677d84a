// Host-side construction of TMA tensor maps.  The driver entry point
// cuTensorMapEncodeTiled is resolved at run time through the CUDA runtime, so
// the library links against nothing but the (static) runtime and loads on a
// machine without a driver.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <mutex>

#include "plan.h"

namespace ts2ts {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  if (fn) return fn;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) != cudaSuccess ||
      qres != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = reinterpret_cast<EncodeTiledFn>(p);
  return fn;
}

// Encoding a map needs a current context, and a thread that has made no CUDA call yet (an autograd worker, say) has none.
inline void bind_context() {
  typedef CUresult (*CtxGetCurrentFn)(CUcontext*);
  static CtxGetCurrentFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess) return;
    fn = reinterpret_cast<CtxGetCurrentFn>(p);
  }
  CUcontext ctx = nullptr;
  int dev = 0;
  if (fn(&ctx) == CUDA_SUCCESS && ctx == nullptr && cudaGetDevice(&dev) == cudaSuccess) cudaSetDevice(dev);
}

// bf16 tensor [B,H,T,D] with D contiguous and element strides (sb, sh, st); tile = `rows` tokens x `cols` elements of one
// (b,h), written to shared memory in columns of 64 elements, one after the other, with the 128-byte swizzle.  Rows past T read as zero and are not written.
// Returns 0 on success.
inline int make_tile_map(CUtensorMap* out, const void* base, int64_t B, int64_t H, int64_t T, int64_t D, int64_t sb, int64_t sh, int64_t st,
                         int rows, int cols) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return -100;
  bind_context();
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0) return -101;
  cuuint64_t dims[5] = {64, (cuuint64_t)T, (cuuint64_t)(D / 64), (cuuint64_t)H, (cuuint64_t)B};
  cuuint64_t strides[4] = {(cuuint64_t)st * 2, 128, (cuuint64_t)sh * 2, (cuuint64_t)sb * 2};
  for (int i = 0; i < 4; ++i)
    if (strides[i] % 16 != 0) return -102;
  cuuint32_t box[5] = {64, (cuuint32_t)rows, (cuuint32_t)(cols / 64), 1, 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -103;
}

// The same map through a small per-process cache: a training step calls the attention entry points once per layer
// with the same few (pointer, shape, strides) combinations, and encoding a map costs a driver call each time.  A key has a set of
// four entries to itself and the few keys that fall on it, so that a look-up compares four keys however many maps are kept: a
// forward and backward asks for twelve, and a program that takes turns between a few sets of buffers keeps all of theirs.
// The map is copied out, so a later request that recycles the cache entry cannot change what a caller holds.
constexpr int kMapSets = 128, kMapWays = 4;
struct MapKey {
  const void* base;
  int64_t v[9];
  int64_t dev;
};
inline int cached_tile_map(CUtensorMap* out, const void* base, int64_t B, int64_t H, int64_t T, int64_t D, int64_t sb, int64_t sh, int64_t st,
                           int rows, int cols) {
  struct Entry { MapKey key; CUtensorMap map; bool used; };
  struct Set { Entry entry[kMapWays]; int next; };
  static Set cache[kMapSets];
  static std::mutex mu;
  int dev = 0;
  cudaGetDevice(&dev);
  const MapKey key = {base, {B, H, T, D, sb, sh, st, rows, cols}, dev};
  uint64_t h = reinterpret_cast<uintptr_t>(base);
  for (int i = 0; i < 9; ++i) h = (h ^ static_cast<uint64_t>(key.v[i])) * 0x9e3779b97f4a7c15ull;
  Set& set = cache[(h ^ (h >> 32) ^ static_cast<uint64_t>(dev)) >> 7 & (kMapSets - 1)];
  std::lock_guard<std::mutex> lock(mu);
  for (Entry& e : set.entry)
    if (e.used && memcmp(&e.key, &key, sizeof(key)) == 0) {
      *out = e.map;
      return 0;
    }
  Entry& e = set.entry[set.next];
  const int r = make_tile_map(&e.map, base, B, H, T, D, sb, sh, st, rows, cols);
  if (r) {
    e.used = false;
    return r;
  }
  e.key = key;
  e.used = true;
  *out = e.map;
  set.next = (set.next + 1) % kMapWays;
  return 0;
}

}  // namespace ts2ts
