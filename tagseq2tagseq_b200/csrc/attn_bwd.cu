// Masked flash-attention backward for sm_100a.
//
// Three kernels:
//   bwd_prep     delta[q] = sum_d O[q,d] dO[q,d],  lse2[q] = LSE[q] * log2(e)   (fp32, side by side for every 32 queries, padded to
//                whole tiles); zeroes dQ
//   attn_bwd     one CTA per 128-key tile of one (batch, head); walks 128-query tiles gathered from the stretches of 32
//                query rows that hold an allowed pair (PlanLayout::bwd_sub; 9-19 % fewer tiles on linked 16k packs, 4-11 % on linked 32k ones; linked 16k,
//                H = 16: D = 128 1004 -> 956 us, H = 12, D = 64 503 -> 471, warm and at the power limit).  Scores are transposed so that a tensor-memory lane is a key row:
//                  tcgen05  S^T = K Q^T,  dP^T = V dO^T            [128 keys x 128 queries, fp32 in TMEM]
//                  warps 0-7 (two threads per key row, 64 queries each), in two phases:
//                           P^T = exp2(scale S^T - lse2[q]) under the mask, as soon as S^T is complete, written as
//                           bf16 over the S^T columns just read; then, once dP^T is complete,
//                           dS^T = P^T (dP^T - delta[q]) as bf16 to shared memory
//                  tcgen05  dV += P^T dO                          (A from TMEM, B MN-major from smem)
//                           S^T of the NEXT tile (D = 128: once dV is complete)
//                           dK += dS^T Q,  dQ = dS K              (dS^T from smem: K-major for dK, MN-major for dQ)
//                           dP^T of the next tile once dQ has been read out of the columns they share
//                  warps 8-11 (thread = query)  dQ -> fp32, 32 head dimensions at a time, through two
//                           private shared-memory boxes per warp -> bulk reduce-adds into the dQ accumulator
//                dV and S^T run while the compute warps form dS^T; dK, dQ and dP^T while they form the exponentials of the
//                next tile (H = 16, linked 16k: 853 -> 794 us at D = 128, 729 -> 600 at D = 64, against a structure with dV and dK behind
//                dS^T).  dK (scaled) and dV leave through shared memory and TMA stores at the end.
//   dq_convert   dQ accumulator (fp32) -> scaled bf16 dq
//
// Computes what the reference gets from autograd of PyTorch FlexAttention
// (torch/_higher_order_ops/flex_attention.py:947-1075): P = exp(S - LSE), dV = P^T dO, dP = dO V^T,
// dS = P (dP - delta), dQ = scale dS K, dK = scale dS^T Q.  Rows whose LSE is -inf get zero gradients.
#include "launch.cuh"
#include "plan.h"
#include "profile.h"
#include "ptx.cuh"
#include "tma_host.h"

#include <math_constants.h>

#include <type_traits>

// A debug build may name a private header that defines the hooks below to record clock64() stamps.
#ifdef TS2TS_BWD_TRACE_HEADER
#include TS2TS_BWD_TRACE_HEADER
#else
#define TS2TS_BWD_TRACE_FIELDS
#define TRACE(role, step, ev) do { } while (0)
#define BTRACE_ACC_DECL
#define BTRACE_ACC(k) do { } while (0)
#define BTRACE_ACC_DUMP() do { } while (0)
#define BTRACE_ATTACH(params, stream) do { } while (0)
#define BTRACE_DUMP(stream) do { } while (0)
#endif

#ifndef TS2TS_BWD_GROUP_MB
// Q/dO bytes of the heads whose CTAs are interleaved in the launch order.  Measured on the 32k masks in the
// seconds-long benchmark loop: 32 MB (one head at 32k, three at 16k) gives the best whole-step rate, 2-3 % above 64 MB
// and 16 MB; 136 MB is 4 % slower and all heads 10 % slower (Q / dO fall out of L2).
#define TS2TS_BWD_GROUP_MB 32
#endif

namespace ts2ts {

struct BwdParams {
  PlanView plan;
  MaskArgs mask;
  const float* stats;    // [B,H,Tp/32][2][32]: -lse2, then -delta
  float* dq_acc;         // [B,H,Tp/32][D/4][32 queries][4], unscaled
  __nv_bfloat16* dk;     // for the empty-list path only
  __nv_bfloat16* dv;
  int64_t dk_s[3], dv_s[3];
  int H, Tp;
  int head_group;        // heads whose CTAs are interleaved in the launch order
  float scale, scale_log2;
  TS2TS_BWD_TRACE_FIELDS
};

constexpr int kBwdThreads = 512;  // warps 0-7 exp/dS, 8-11 dQ reduction, 12 and 14 TMA producers, 13 MMA issuer, 15 idle
constexpr int kSubQ = 64;         // query columns per compute half

template <int D>
struct BwdSmem {
  static constexpr int kSub = D / 64;
  static constexpr int kTileBytes = kTile * D * 2;
  static constexpr int kDsBytes = kTile * kTile * 2;  // dS^T: two halves of [128 key rows x 128 B]
  static constexpr int kQStages = D == 64 ? 3 : 2, kDoStages = D == 64 ? 2 : 1;  // what shared memory holds
  static constexpr int kSBufs = D == 64 ? 2 : 1;       // S^T buffers: what tensor memory holds
  static constexpr int kStageBytes = 4 * 2 * 4096;     // dQ staging: per reduction warp two boxes of 32 queries x 32 floats
  // K, V, Q stages, dO buffers, dS^T, the dQ staging boxes, then row statistics, barriers and flags; plus
  // alignment slack.  The kernel declares no static shared memory, so the dynamic region normally starts 1024-byte
  // aligned and the slack stays unused; if it ever does not fit, the kernel reports status 2900 instead of running.
  static constexpr int kTiles = (2 + kQStages + kDoStages) * kTileBytes + kDsBytes + kStageBytes;
  static constexpr int kTileSlots = 4;  // a tile's stretch numbers outlive its Q stage until dQ has been read out: one more slot than stages
  static constexpr int kStats = 2 * kQStages * kTile * 4, kBars = 20;
  static constexpr int kSmall = kStats + kBars * 8 + 16 + kQStages * kMaskRuns * 16 + kTileSlots * 8;  // statistics, barriers, flags, staged masks and stretch numbers
  static constexpr int kSlack = 512;
  static constexpr int kBytes = kTiles + kSmall + kSlack;
  // tensor-memory columns: dV, dK accumulators, S^T (later P^T), dP^T (later dQ)
  static constexpr int kDV = 0, kDK = D, kST = 2 * D, kDPT = 2 * D + 128 * kSBufs;
};

template <uint32_t N> __device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <uint32_t N> __device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// A query tile as the kernel walks them: the numbers of four stretches of 32 query rows, kStretchFull set in a full tile
// (PlanLayout::bwd_sub).  Sequences beyond the table walk whole q tiles.
__device__ __forceinline__ uint32_t stretch_entry(const uint16_t* subs, const int32_t* list, int i, int j, int NB) {
  if (subs != nullptr) {
    uint16_t v;
    asm volatile("ld.global.nc.b16 %0, [%1];" : "=h"(v) : "l"(subs + kStretches * i + j));
    return v;
  }
  const int entry = ld_nc_i32_here(list + i);
  return kStretches * min(static_cast<int>(entry & ~kFullBit), NB - 1) + j | ((entry & kFullBit) ? kStretchFull : 0u);
}
// Stretch number of an entry; kStretches * NB stands for no stretch.
__device__ __forceinline__ int stretch_of(uint32_t entry, int NB) { return min(static_cast<int>(entry & ~kStretchFull), kStretches * NB); }

// Masks of the query rows of two stretches (the numbers in `pair`) that may read key `row` of tile kb, before causality, from
// the run lists: the way out for keys that the plan's mask table does not cover (see kMaskRuns).  "May row class r read my
// column class" is looked up in the transposed table where the pre-pass built one.
__device__ __noinline__ uint2 key_masks(const PlanView& P, const MaskArgs& M, int b, uint32_t pair, int kb, int row) {
  const int kv = kb * kTile + row;
  if (kv >= P.T) return make_uint2(0u, 0u);
  const int kvdoc = M.doc[(size_t)b * P.T + kv], kvcol = M.col[(size_t)b * P.T + kv];
  const bool linked = M.link != nullptr && kvcol >= 0 && kvcol < 64 * M.W;
  const unsigned long long* lt_row = nullptr;
  const int64_t* link_col = nullptr;
  if (linked && P.status[kLinkTRows] == M.R && kvcol < kLinkTMaxCols) lt_row = P.link_t + ((size_t)b * kLinkTMaxCols + kvcol) * kLinkTWords;
  else if (linked) link_col = M.link + (size_t)b * M.R * M.W + (kvcol >> 6);
  uint32_t bits[2] = {0u, 0u};
#pragma unroll 1
  for (int s = 0; s < 2; ++s) {
    const int sub = stretch_of(pair >> (16 * s) & 0xffffu, P.NB);
    if (sub == kStretches * P.NB) continue;
    const int qb = sub / kStretches, from = sub % kStretches * kStretch;
    const size_t tq = (size_t)b * P.NB + qb;
    const int4* runs = reinterpret_cast<const int4*>(P.runs + tq * kTile);
    const int n = min(__ldg(&P.run_cnt[tq]), kTile), n_valid = min(kTile, P.T - qb * kTile);
    uint32_t mask = 0u;
    int4 cur = __ldg(runs);
    for (int r = 0; r < n && cur.x < from + kStretch; ++r) {
      const int4 nx = r + 1 < n ? __ldg(runs + r + 1) : make_int4(n_valid, 0, 0, 0);
      const int lo = max(cur.x - from, 0), hi = min(nx.x - from, kStretch);  // the run covers these rows of the stretch
      if (hi > lo) {
        bool allowed = cur.y == kvdoc;
        if (!allowed && linked && cur.z >= 0 && cur.z < M.R)
          allowed = lt_row != nullptr ? (__ldg(lt_row + (cur.z >> 6)) >> (cur.z & 63)) & 1ull
                                      : (static_cast<unsigned long long>(__ldg(link_col + (size_t)cur.z * M.W)) >> (kvcol & 63)) & 1ull;
        if (allowed) mask |= (0xffffffffu >> (kStretch - (hi - lo))) << lo;
      }
      cur = nx;
    }
    if (s == 0) bits[0] = mask; else bits[1] = mask;
  }
  return make_uint2(bits[0], bits[1]);
}

// The per-tile arithmetic of a compute thread, 32 query columns at a time, in two phases so that the first can run
// while the tensor core still works on dK and dQ of the previous tile and dP^T of this one:
//   p_chunk   P^T = exp2(scale S^T - lse2) under the mask, packed to bf16 pairs (the MMA operand, also kept in
//             registers for the second phase)
//   ds_chunk  dS^T = P^T (dP^T - delta), from the bf16 P^T, packed to bf16 pairs
// The row statistics of the 32 queries are read from shared memory; every lane of a warp reads the same addresses.
// `nl2` / `ndl` hold the NEGATED statistics (-lse2, -delta), so that both phases are one packed multiply-add /
// add per two queries (fp32x2 instructions; a 16-byte shared-memory load yields two ready operand pairs).
template <bool kMasked>
__device__ __forceinline__ void p_body(const uint32_t (&s)[32], const float* nl2, uint32_t bw, float scale_log2, uint32_t (&pk)[16]) {
  const unsigned long long scale2 = pack_f32x2(scale_log2, scale_log2);
#pragma unroll
  for (int e = 0; e < 32; e += 4) {
    const ulonglong2 n4 = *reinterpret_cast<const ulonglong2*>(nl2 + e);
    float x0, x1, x2, x3;
    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(s[e + 0]), __uint_as_float(s[e + 1])), scale2, n4.x), x0, x1);
    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(s[e + 2]), __uint_as_float(s[e + 3])), scale2, n4.y), x2, x3);
    float p0 = fast_exp2(x0), p1 = fast_exp2(x1), p2 = fast_exp2(x2), p3 = fast_exp2(x3);
    if (kMasked) {
      p0 = ((bw >> (e + 0)) & 1u) ? p0 : 0.f;
      p1 = ((bw >> (e + 1)) & 1u) ? p1 : 0.f;
      p2 = ((bw >> (e + 2)) & 1u) ? p2 : 0.f;
      p3 = ((bw >> (e + 3)) & 1u) ? p3 : 0.f;
    }
    pk[(e >> 1) + 0] = pack_bf16(p0, p1);
    pk[(e >> 1) + 1] = pack_bf16(p2, p3);
  }
}
// mode: 0 = every query allowed, 1 = test the bits of `bw`, 2 = no query allowed (nothing is computed).  kMasked = false is
// the code of full tiles, which knows no modes.
template <bool kMasked>
__device__ __forceinline__ void p_chunk(const uint32_t (&s)[32], const float* nl2, uint32_t bw, int mode, float scale_log2,
                                        uint32_t (&pk)[16]) {
  if (!kMasked || mode == 0) {
    p_body<false>(s, nl2, bw, scale_log2, pk);
  } else if (mode == 1) {
    p_body<true>(s, nl2, bw, scale_log2, pk);
  } else {
#pragma unroll
    for (int e = 0; e < 16; ++e) pk[e] = 0u;
  }
}
template <bool kMasked>
__device__ __forceinline__ void ds_chunk(const uint32_t (&pk)[16], const uint32_t (&dp)[32], const float* ndl, int mode,
                                         uint32_t (&dsk)[16]) {
  if (kMasked && mode == 2) {
#pragma unroll
    for (int e = 0; e < 16; ++e) dsk[e] = 0u;
    return;
  }
#pragma unroll
  for (int e = 0; e < 32; e += 4) {
    const ulonglong2 d4 = *reinterpret_cast<const ulonglong2*>(ndl + e);
    const uint32_t a = pk[(e >> 1) + 0], c = pk[(e >> 1) + 1];
    const unsigned long long p01 = pack_f32x2(__uint_as_float(a << 16), __uint_as_float(a & 0xffff0000u));
    const unsigned long long p23 = pack_f32x2(__uint_as_float(c << 16), __uint_as_float(c & 0xffff0000u));
    float r0, r1, r2, r3;
    unpack_f32x2(mul_f32x2(p01, add_f32x2(pack_f32x2(__uint_as_float(dp[e + 0]), __uint_as_float(dp[e + 1])), d4.x)), r0, r1);
    unpack_f32x2(mul_f32x2(p23, add_f32x2(pack_f32x2(__uint_as_float(dp[e + 2]), __uint_as_float(dp[e + 3])), d4.y)), r2, r3);
    dsk[(e >> 1) + 0] = pack_bf16(r0, r1);
    dsk[(e >> 1) + 1] = pack_bf16(r2, r3);
  }
}

template <int D>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapDO,
                const __grid_constant__ CUtensorMap mapQs, const __grid_constant__ CUtensorMap mapDOs,
                const __grid_constant__ CUtensorMap mapDK, const __grid_constant__ CUtensorMap mapDV,
                const __grid_constant__ BwdParams p) {
  using Cfg = BwdSmem<D>;
  extern __shared__ uint8_t smem_raw[];
  // Plain pointer arithmetic (no round trip through an integer) keeps the shared address space visible to the
  // compiler, so every access below becomes a shared-memory instruction instead of a generic one.
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sK = smem;
  uint8_t* sV = smem + Cfg::kTileBytes;
  uint8_t* sQ = smem + 2 * Cfg::kTileBytes;       // Cfg::kQStages stages
  uint8_t* sDO = sQ + Cfg::kQStages * Cfg::kTileBytes;  // Cfg::kDoStages buffers
  uint8_t* sDS = sDO + Cfg::kDoStages * Cfg::kTileBytes;  // dS^T, halves of 16 KB
  uint8_t* sStage = sDS + Cfg::kDsBytes;          // dQ staging boxes
  float* s_stats = reinterpret_cast<float*>(smem + Cfg::kTiles);  // [Q stages][kStretches][2][32]: -lse2, then -delta
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kTiles + Cfg::kStats);
  uint64_t& bar_kv = bars[0];
  uint64_t* bar_q_full = bars + 1;     // [Q stages] Q, lse2, delta of a stage landed
  uint64_t* bar_do_full = bars + 4;    // [dO buffers] dO of the tile landed
  uint64_t* bar_gv = bars + 6;         // [dO buffers] dV MMAs of the tile completed: its dO buffer may be reloaded
  uint64_t* bar_gq = bars + 8;         // [Q stages] dK MMAs of the tile completed: its Q stage may be reloaded
  uint64_t* bar_s = bars + 11;         // [S^T buffers] S^T of the tile is in tensor memory
  uint64_t* bar_p = bars + 13;         // [tile & 1] P^T written
  uint64_t& bar_dp = bars[15];         // dP^T of the tile is in tensor memory
  uint64_t& bar_ds = bars[16];         // dS^T written
  uint64_t& bar_g = bars[17];          // dQ of the tile is in tensor memory
  uint64_t& bar_dqr = bars[18];        // dQ read out of tensor memory
  uint64_t& bar_epi = bars[19];
  uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + Cfg::kBars);
  volatile int* abort_ptr = reinterpret_cast<volatile int*>(reinterpret_cast<uint8_t*>(bars + Cfg::kBars) + 4);
  int* abort_w = const_cast<int*>(abort_ptr);
  uint32_t* s_masks = reinterpret_cast<uint32_t*>(bars + Cfg::kBars + 2);  // [Q stages][kStretches][kMaskRuns] the tile's masks, by run of the key
  uint32_t* s_tile = s_masks + Cfg::kQStages * kStretches * kMaskRuns;  // [kTileSlots][2] a tile's four stretch entries, 16 bits each
  static_assert(Cfg::kTileSlots > Cfg::kQStages, "");
  if (smem + Cfg::kTiles + Cfg::kSmall > smem_raw + Cfg::kBytes) {  // a misplaced shared-memory window, the same in all CTAs: refused before anything is written there
    if (threadIdx.x == 0) atomicCAS(p.plan.status, 0, 2900);
    wait_previous();
    return;
  }

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const PlanView& P = p.plan;
  const int NB = P.NB;
  // Launch order (the hardware starts CTAs by ascending blockIdx): batch elements one after the other; inside one,
  // groups of G heads; inside a group all heads' heaviest kv tiles first, then their second heaviest, and so on.  The
  // group bounds the Q / dO working set that has to stay in L2, and the long CTAs of the last group still start well
  // before the end of the launch instead of running alone at its tail.
  const int per_b = p.H * NB, G = p.head_group;
  const int b = blockIdx.x / per_b;
  const int r1 = blockIdx.x - b * per_b;
  const int grp = r1 / (G * NB);
  const int r2 = r1 - grp * G * NB;
  const int gsize = min(G, p.H - grp * G);
  const int rank = r2 / gsize;
  const int h = grp * G + (r2 - rank * gsize);
  // What the plan says is under way while the barriers and the tensor memory are set up; inside the plan's buffer whatever it holds.
  const int magic = ld_nc_i32_here(P.status + kStampMagic), plan_b = ld_nc_i32_here(P.status + kStampB), plan_t = ld_nc_i32_here(P.status + kStampT);
  const int place = ld_nc_i32_here(P.bwd_order + (size_t)b * NB + rank);

  if (tid == 0) {
    *abort_ptr = 0;
    mbar_init(&bar_kv, 2);
    for (int i = 0; i < 3; ++i) {
      mbar_init(&bar_q_full[i], 1);
      mbar_init(&bar_gq[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_do_full[i], 1);
      mbar_init(&bar_gv[i], 1);
      mbar_init(&bar_s[i], 1);
      mbar_init(&bar_p[i], 8);  // one arrival per compute warp
    }
    mbar_init(&bar_dp, 1);
    mbar_init(&bar_ds, 8);
    mbar_init(&bar_g, 1);
    mbar_init(&bar_dqr, 4);  // one arrival per reduction warp
    mbar_init(&bar_epi, 8);
    fence_mbar_init();
  }
  __syncthreads();
  if (warp == 13) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  const int kb = min(max(place, 0), NB - 1);
  const int tiles = ld_nc_i32_here((P.bwd_sub != nullptr ? P.bwd_tiles : P.bwd_cnt) + (size_t)b * NB + kb);
  const int32_t* list = P.bwd_idx + ((size_t)b * NB + kb) * NB;
  const uint16_t* subs = P.bwd_sub != nullptr ? P.bwd_sub + ((size_t)b * sub_line(NB, NB) + sub_line(NB, kb)) * kStretches : nullptr;
  uint32_t entry = 0u;  // the producers' first one
  if (warp == 12 || warp == 14) entry = stretch_entry(subs, list, 0, lane & (kStretches - 1), NB);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const int n = min(max(tiles, 0), NB - kb);  // query tiles to walk
  const bool bad = magic != kPlanMagic || plan_b != P.B || plan_t != P.T;  // uniform across the grid: refuse a plan that was not built for this (B, T)
  if (bad || n == 0) {
    if (bad) {
      if (tid == 0) atomicCAS(P.status, 0, 2901);
    } else if (tid < kTile) {
      const int kv = kb * kTile + tid;
      if (kv < P.T) {
        __nv_bfloat16* a = p.dk + (size_t)b * p.dk_s[0] + (size_t)h * p.dk_s[1] + (size_t)kv * p.dk_s[2];
        __nv_bfloat16* c = p.dv + (size_t)b * p.dv_s[0] + (size_t)h * p.dv_s[1] + (size_t)kv * p.dv_s[2];
        for (int i = 0; i < D; i += 8) {
          *reinterpret_cast<uint4*>(a + i) = make_uint4(0, 0, 0, 0);
          *reinterpret_cast<uint4*>(c + i) = make_uint4(0, 0, 0, 0);
        }
      }
    }
    if (warp == 13) tmem_dealloc(tmem, 512);
    wait_previous();
    return;
  }
  const uint32_t tDV = tmem + Cfg::kDV, tDK = tmem + Cfg::kDK, tST = tmem + Cfg::kST, tDPT = tmem + Cfg::kDPT, tDQ = tDPT;
  // S^T columns [32c, +32) of a buffer are read by the compute thread of (row, c / 2), which writes P^T bf16 over the first 16 of them.

  if (warp >= 12) {
    if (D == 64) reg_dec<112>(); else reg_dec<88>();
    if (warp == 12 || warp == 14) {
      // ---------------------------------------------------------------- TMA producers: warp 12 K and Q, warp 14 V and dO
      // A q tile as it lies in memory comes in one box; a gathered one by a lane each for its stretches, in boxes of 32 rows.  A
      // stretch past the sequence reads as zeros, has no statistics and no masks, and nothing is computed from it.  Every
      // copy takes its issuing thread 100-150 clk, and a tile's first product waits for the last of them.
      const bool is_q = warp == 12, mine = lane < kStretches;
      const CUtensorMap *whole = is_q ? &mapQ : &mapDO, *part = is_q ? &mapQs : &mapDOs;
      if (lane == 0) {
        const CUtensorMap* kv = is_q ? &mapK : &mapV;
        tma_prefetch_desc(kv); tma_prefetch_desc(whole); tma_prefetch_desc(part);
        mbar_expect_tx(&bar_kv, Cfg::kTileBytes);
        tma_load_tile(is_q ? sK : sV, kv, &bar_kv, kb * kTile, 0, h, b);
      }
      wait_previous();  // the row statistics; dQ's zeros, which everything that adds to them comes after
      const float* stats = p.stats + ((size_t)b * p.H + h) * p.Tp * 2;
      const uint32_t* masks = P.kv_mask + (size_t)b * ((size_t)NB * (NB + 1) / 2) * (kStretches * kMaskRuns);
      const int stages = is_q ? Cfg::kQStages : Cfg::kDoStages;
      uint8_t* tiles = is_q ? sQ : sDO;
      uint64_t *full = is_q ? bar_q_full : bar_do_full, *free = is_q ? bar_gq : bar_gv;
      int st = 0, use = 0;
      for (int i = 0; i < n; ++i) {
        const int sub = stretch_of(entry, NB);
        const uint32_t next = i + 1 < n ? stretch_entry(subs, list, i + 1, lane & (kStretches - 1), NB) : 0u;
        const int first = __shfl_sync(0xffffffffu, sub, 0);
        const bool joined = __all_sync(0xffffffffu, sub == first + (lane & (kStretches - 1)) && sub < kStretches * NB) && first % kStretches == 0;
        const bool live = mine && sub < kStretches * NB, masked = !(entry & kStretchFull) && P.kv_mask != nullptr;
        const uint32_t n_live = __popc(__ballot_sync(0xffffffffu, live));
        if (use > 0 && !mbar_wait_warp(&free[st], (use - 1) & 1, abort_w, is_q ? 12 : 11)) break;  // dK / dV MMAs of the tile before done
        if (is_q && mine) reinterpret_cast<uint16_t*>(s_tile)[(i % Cfg::kTileSlots) * kStretches + lane] = entry;
        __syncwarp();
        if (lane == 0) mbar_expect_tx(&full[st], Cfg::kTileBytes + (is_q ? n_live * (2 * kStretch * 4 + (masked ? kMaskRuns * 4 : 0)) : 0u));
        __syncwarp();
        uint8_t* dst = tiles + st * Cfg::kTileBytes;
        float* stat = s_stats + st * (2 * kTile) + lane * (2 * kStretch);
        uint32_t* mask = s_masks + (st * kStretches + lane) * kMaskRuns;
        const uint32_t* mask_src = masks + (mask_pair(sub / kStretches, kb) * kStretches + sub % kStretches) * kMaskRuns;
        if (joined) {
          if (lane == 0) {
            tma_load_tile(dst, whole, &full[st], sub * kStretch, 0, h, b);
            if (is_q) bulk_load(stat, stats + sub * (2 * kStretch), 2 * kTile * 4, &full[st]);
            if (is_q && masked) bulk_load(mask, mask_src, kStretches * kMaskRuns * 4, &full[st]);
          }
        } else if (mine) {
          for (int s = 0; s < Cfg::kSub; ++s) tma_load_tile(dst + s * 16384 + lane * (kStretch * 128), part, &full[st], sub * kStretch, s, h, b);
          if (is_q && live) {
            bulk_load(stat, stats + sub * (2 * kStretch), 2 * kStretch * 4, &full[st]);
            if (masked) bulk_load(mask, mask_src, kMaskRuns * 4, &full[st]);
          }
        }
        entry = next;
        if (++st == stages) { st = 0; ++use; }
      }
    } else if (warp == 13 && lane == 0) {
      // ---------------------------------------------------------------- MMA issuer
      constexpr uint32_t idesc_st = make_idesc_bf16(128, 128, false, false);  // K-major x K-major
      constexpr uint32_t idesc_g = make_idesc_bf16(128, D, false, true);      // TMEM or K-major A x MN-major B, N = D
      constexpr uint32_t idesc_dq = make_idesc_bf16(128, D, true, true);      // MN-major A x MN-major B, N = D
      // Descriptor halves (see desc_lo / desc_hi): `hi` is shared by every operand (SBO = 1024); K-major operands
      // carry LBO 16, MN-major ones LBO 16384 (distance between the two 64-element halves of the MN extent).
      constexpr uint32_t hi = desc_hi(1024);
      constexpr uint32_t kTileStep = Cfg::kTileBytes >> 4;
      const uint32_t k_kmaj = desc_lo(smem_u32(sK), 16), v_kmaj = desc_lo(smem_u32(sV), 16);
      const uint32_t q_kmaj = desc_lo(smem_u32(sQ), 16), do_kmaj = desc_lo(smem_u32(sDO), 16), ds_kmaj = desc_lo(smem_u32(sDS), 16);
      const uint32_t q_mn = desc_lo(smem_u32(sQ), 16384), do_mn = desc_lo(smem_u32(sDO), 16384);
      const uint32_t k_mn = desc_lo(smem_u32(sK), 16384), ds_mn = desc_lo(smem_u32(sDS), 16384);
      auto kstep = [](int kk) -> uint32_t { return ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4; };  // 16 elements along a K-major operand
      // Shared-memory accesses of this thread (barrier waits included) queue behind the MMAs it has issued and only
      // proceed once the tensor pipe has accepted those.  So a group asks, two MMAs before its end, whether what the
      // next group waits for has arrived already (`early`): the pipe stays fed while the answer comes.  dK does not ask: at D = 128 dQ
      // follows, which waits for nothing more, and at D = 64, where dK is the last group, the question for dO comes behind it; the next
      // group there waits for dQ to be read out in any case, and dO has two buffers.
      bool early_p = false, early_q = false, early_ds = false, early_do = false;
      auto q_full = [&](int i) { return mbar_test_wait(&bar_q_full[i % Cfg::kQStages], (i / Cfg::kQStages) & 1); };
      auto do_full = [&](int i) { return mbar_test_wait(&bar_do_full[i % Cfg::kDoStages], (i / Cfg::kDoStages) & 1); };
      auto wait_q = [&](int i) { return early_q || mbar_wait(&bar_q_full[i % Cfg::kQStages], (i / Cfg::kQStages) & 1, abort_w, 22); };
      auto wait_do = [&](int i) { return early_do || mbar_wait(&bar_do_full[i % Cfg::kDoStages], (i / Cfg::kDoStages) & 1, abort_w, 27); };
      auto issue_st = [&](int i, auto ask) {  // S^T = K Q^T
        const uint32_t q = q_kmaj + (i % Cfg::kQStages) * kTileStep, t = tST + (i % Cfg::kSBufs) * 128;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          if (kk == D / 16 - 2) ask();
          mma_ss2(t, k_kmaj + kstep(kk), hi, q + kstep(kk), hi, idesc_st, kk > 0);
        }
        mma_commit(&bar_s[i % Cfg::kSBufs]);
      };
      auto issue_dpt = [&](int i, auto ask) {  // dP^T = V dO^T
        const uint32_t o = do_kmaj + (i % Cfg::kDoStages) * kTileStep;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          if (kk == D / 16 - 2) ask();
          mma_ss2(tDPT, v_kmaj + kstep(kk), hi, o + kstep(kk), hi, idesc_st, kk > 0);
        }
        mma_commit(&bar_dp);
      };
      auto issue_dq = [&](auto ask) {  // dQ = dS K
#pragma unroll
        for (int kk = 0; kk < kTile / 16; ++kk) {
          if (kk == kTile / 16 - 2) ask();
          mma_ss2(tDQ, ds_mn + kk * 128, hi, k_mn + kk * 128, hi, idesc_dq, kk > 0);
        }
        mma_commit(&bar_g);
      };
      auto issue_dk = [&](int i) {  // dK += dS^T Q
        const uint32_t q = q_mn + (i % Cfg::kQStages) * kTileStep;
#pragma unroll
        for (int kk = 0; kk < kTile / 16; ++kk) mma_ss2(tDK, ds_kmaj + kstep(kk), hi, q + kk * 128, hi, idesc_g, (i > 0 || kk > 0) ? 1u : 0u);
        mma_commit(&bar_gq[i % Cfg::kQStages]);
      };
      auto issue_dv = [&](int i, auto ask) {  // dV += P^T dO
        const uint32_t o = do_mn + (i % Cfg::kDoStages) * kTileStep, t = tST + (i % Cfg::kSBufs) * 128;
#pragma unroll
        for (int kk = 0; kk < kTile / 16; ++kk) {
          if (kk == kTile / 16 - 2) ask();
          mma_ts2(tDV, t + (kk >> 1) * 32 + (kk & 1) * 8, o + kk * 128, hi, idesc_g, (i > 0 || kk > 0) ? 1u : 0u);
        }
        mma_commit(&bar_gv[i % Cfg::kDoStages]);
      };
      auto nothing = []() {};
      // Order per tile: dV(i), S^T(i+1) (the other way round where S^T has two buffers) | dK(i), dQ(i) | dP^T(i+1).
      // dV and S^T run while the compute warps work on dS^T(i); dK, dQ and dP^T(i+1) while they work on the exponentials
      // of tile i+1, so both sides always have a phase's worth of work in hand.  With one buffer S^T(i+1) overwrites the
      // P^T columns of tile i and waits for dV(i), which reads them: PTX promises the order of issue only to MMAs with the same
      // accumulator and shape (linked 16k 815 -> 826 us, causal 4k batch 4 650 -> 652).  With two the last reader, dV(i-1), completed
      // before dQ(i-1) was read out.  At D = 64 dQ comes before dK, which then runs while dQ is read out (linked 16k, H = 12: 471 -> 454 us,
      // causal 4k batch 4, H = 16: 531 -> 510).  At D = 128, with two Q stages, dK comes first: the stage it frees is asked for before
      // the copy engine is taken up by dQ's reductions, behind which the next but one tile's Q lands too late (dQ first: 978 -> 1019 us).
      bool ok = mbar_wait(&bar_kv, 0, abort_w, 21) && wait_q(0);
      if (ok) {
        tc_fence_after();
        issue_st(0, nothing);
        ok = wait_do(0);
        if (ok) issue_dpt(0, nothing);
      }
      for (int i = 0; i < n && ok; ++i) {
        const bool more = i + 1 < n;
        TRACE(0, i, 0);
        if (Cfg::kSBufs == 2 && more) {
          if (!(ok = wait_q(i + 1))) break;
          tc_fence_after();
          issue_st(i + 1, [&]() { early_p = mbar_test_wait(&bar_p[i & 1], (i >> 1) & 1); });
        }
        if (!(ok = early_p || mbar_wait(&bar_p[i & 1], (i >> 1) & 1, abort_w, 24))) break;
        tc_fence_after();
        TRACE(0, i, 1);
        issue_dv(i, [&]() {
          if (Cfg::kSBufs == 2) early_ds = mbar_test_wait(&bar_ds, i & 1);
          else early_q = more && q_full(i + 1);
        });
        if (Cfg::kSBufs == 1 && more) {
          if (!(ok = wait_q(i + 1) && mbar_wait(&bar_gv[i % Cfg::kDoStages], (i / Cfg::kDoStages) & 1, abort_w, 29))) break;
          tc_fence_after();
          TRACE(0, i, 2);
          issue_st(i + 1, [&]() { early_ds = mbar_test_wait(&bar_ds, i & 1); });
        }
        TRACE(0, i, 3);
        if (!(ok = early_ds || mbar_wait(&bar_ds, i & 1, abort_w, 28))) break;
        tc_fence_after();
        TRACE(0, i, 4);
        if (D == 64) {
          issue_dq(nothing);
          issue_dk(i);
          early_do = more && do_full(i + 1);
        } else {
          issue_dk(i);
          issue_dq([&]() { early_do = more && do_full(i + 1); });
        }
        TRACE(0, i, 5);
        early_p = early_q = early_ds = false;
        if (more) {
          if (!(ok = wait_do(i + 1) && mbar_wait(&bar_dqr, i & 1, abort_w, 23))) break;  // dQ(i) read out of the columns dP^T(i+1) overwrites
          tc_fence_after();
          TRACE(0, i, 6);
          issue_dpt(i + 1, [&]() {
            if (Cfg::kSBufs == 2) early_q = i + 2 < n && q_full(i + 2);
            else early_p = mbar_test_wait(&bar_p[(i + 1) & 1], ((i + 1) >> 1) & 1);
          });
        }
        early_do = false;
        TRACE(0, i, 7);
      }
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ exp / dS warps: thread = (key row, 64 of the tile's 128 queries)
    // register pool: 256 x 128 (the launch value) + 128 x 168 + 128 x 88 = 512 x 128; at D = 64, where the reduction warps hold
    // half as much, 256 x 120 + 128 x 136 + 128 x 112 (linked 16k 613 -> 600 us: no spills)
    if (D == 64) reg_dec<120>();
    const int row = tid & (kTile - 1), half = tid >> 7;
    const int kv = kb * kTile + row;
    const bool kv_valid = kv < P.T;
    int run = kMaskRuns;  // this key's row of the mask table: the number of its run inside the tile
    if (P.kv_mask != nullptr) {
      const size_t tk = (size_t)b * NB + kb;
      const int nr = __ldg(&P.run_cnt[tk]);
#pragma unroll
      for (int r = 0; r < kMaskRuns + 1; ++r)
        if (r < nr && __ldg(&P.runs[tk * kTile + r].start) <= row) run = r;
    }
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    bool ok = true;
    BTRACE_ACC_DECL
    for (int i = 0; i < n && ok; ++i) {
      const int st = i % Cfg::kQStages;
      if (!(ok = mbar_wait_warp(&bar_q_full[st], (i / Cfg::kQStages) & 1, abort_w, 30))) break;  // Q, -lse2, -delta, the masks and the stretch numbers of this tile landed
      // Full and partial tiles are separate code: the full one carries no mask state, so that its two phases fit the
      // registers and the instruction cache (first phase 2080 -> 1500 clk a tile, causal 4k, D = 128).
      auto tile = [&](auto masked_tag) {
        constexpr bool kMasked = decltype(masked_tag)::value;
        // per 32-query chunk of this thread, uniform over the warp: 0 all allowed, 1 test bits, 2 nothing allowed
        int mode[2] = {0, 0};
        uint32_t bw[2] = {0xffffffffu, 0xffffffffu};
        if (kMasked) {
          const uint32_t mine = s_tile[i % Cfg::kTileSlots * 2 + half];  // this thread's two stretches
          if (run < kMaskRuns) {
            const uint32_t* m = s_masks + (st * kStretches + 2 * half) * kMaskRuns + run;
            bw[0] = m[0]; bw[1] = m[kMaskRuns];
          } else {
            const uint2 m2 = key_masks(P, p.mask, b, mine, kb, row);
            bw[0] = m2.x; bw[1] = m2.y;
          }
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const uint32_t entry = mine >> (16 * s) & 0xffffu;
            const int sub = stretch_of(entry, NB), lo = row - sub % kStretches * kStretch;
            if (sub / kStretches == kb)  // causal inside the diagonal tile: query rows row..127
              bw[s] &= lo <= 0 ? 0xffffffffu : (lo >= 32 ? 0u : ~((1u << lo) - 1u));
            if (!kv_valid || sub == kStretches * NB) bw[s] = 0u;
            mode[s] = __all_sync(0xffffffffu, bw[s] == 0u) ? 2 : (__all_sync(0xffffffffu, bw[s] == 0xffffffffu) ? 0 : 1);
          }
        }
        if (kMasked) BTRACE_ACC(0); else BTRACE_ACC(1);
        // ---- phase 1: exponentials, as soon as S^T is complete, 32 columns at a time (the second load in
        //      flight behind the first half's arithmetic takes registers that spill: 3960 -> 4120 clk a tile)
        if (!mbar_wait_warp(&bar_s[i % Cfg::kSBufs], (i / Cfg::kSBufs) & 1, abort_w, 35)) return false;
        tc_fence_after();
        BTRACE_ACC(2);
        if ((tid & 127) == 0) TRACE(1 + half, i, 0);
        const uint32_t tSc = tST + (i % Cfg::kSBufs) * 128 + lane_base + 64 * half;
        const float* stats = s_stats + st * (2 * kTile) + half * (2 * kSubQ);
        uint32_t pk[2][16];
        {
          uint32_t s0[32], s1[32];
          tmem_ld32(tSc, s0);
          tmem_ld_wait();
          p_chunk<kMasked>(s0, stats, bw[0], mode[0], p.scale_log2, pk[0]);
          tmem_st16(tSc, pk[0]);
          tmem_ld32(tSc + 32, s1);
          tmem_ld_wait();
          p_chunk<kMasked>(s1, stats + 2 * kStretch, bw[1], mode[1], p.scale_log2, pk[1]);
          tmem_st16(tSc + 32, pk[1]);
          tmem_st_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_p[i & 1]);
        if ((tid & 127) == 0) TRACE(1 + half, i, 1);
        BTRACE_ACC(3);
        // ---- phase 2: dS^T, once dP^T is complete.  dP^T(i) was issued after the MMAs that read dS^T(i-1), so its buffer
        // is free as well.
        if (!mbar_wait_warp(&bar_dp, i & 1, abort_w, 31)) return false;
        tc_fence_after();
        BTRACE_ACC(4);
        if ((tid & 127) == 0) TRACE(1 + half, i, 2);
        {
          const uint32_t tDc = tDPT + lane_base + 64 * half;
          uint8_t* ds_row = sDS + half * 16384;  // row `row`: 64 queries, 128 bytes
          uint32_t d0[32], d1[32], dsk[16];
          tmem_ld32(tDc, d0);
          tmem_ld_wait();
          ds_chunk<kMasked>(pk[0], d0, stats + kStretch, mode[0], dsk);
#pragma unroll
          for (int g = 0; g < 4; ++g)
            *reinterpret_cast<uint4*>(ds_row + sw128_offset(row, g)) = make_uint4(dsk[g * 4 + 0], dsk[g * 4 + 1], dsk[g * 4 + 2], dsk[g * 4 + 3]);
          tmem_ld32(tDc + 32, d1);
          tmem_ld_wait();
          ds_chunk<kMasked>(pk[1], d1, stats + 3 * kStretch, mode[1], dsk);
#pragma unroll
          for (int g = 0; g < 4; ++g)
            *reinterpret_cast<uint4*>(ds_row + sw128_offset(row, 4 + g)) = make_uint4(dsk[g * 4 + 0], dsk[g * 4 + 1], dsk[g * 4 + 2], dsk[g * 4 + 3]);
        }
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_ds);
        if ((tid & 127) == 0) TRACE(1 + half, i, 3);
        return true;
      };
      ok = (s_tile[i % Cfg::kTileSlots * 2] & kStretchFull) ? tile(std::false_type{}) : tile(std::true_type{});
      if (!ok) break;
      BTRACE_ACC(5);
    }
    // ---- epilogue: dV (query-half 0 threads) and scale * dK (half 1) -> bf16 -> swizzled smem -> TMA stores.
    //      dV goes through the Q stage the last tile did not use, dK through a dO buffer; what read
    //      them, and the MMAs that add to dV and dK, completed before bar_gq.
    const int est = n % Cfg::kQStages;
    if (ok) ok = mbar_wait_warp(&bar_gq[(n - 1) % Cfg::kQStages], ((n - 1) / Cfg::kQStages) & 1, abort_w, 32);
    tc_fence_after();
    uint8_t* out_dv = sQ + est * Cfg::kTileBytes;
    uint8_t* out_dk = sDO;
    if (ok) {
      const uint32_t tsrc = half == 0 ? tDV : tDK;
      uint8_t* stage = half == 0 ? out_dv : out_dk;
      const float f = half == 0 ? 1.f : p.scale;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t r[32];
        tmem_ld32(tsrc + lane_base + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 v;
          v.x = pack_bf16(__uint_as_float(r[g * 8 + 0]) * f, __uint_as_float(r[g * 8 + 1]) * f);
          v.y = pack_bf16(__uint_as_float(r[g * 8 + 2]) * f, __uint_as_float(r[g * 8 + 3]) * f);
          v.z = pack_bf16(__uint_as_float(r[g * 8 + 4]) * f, __uint_as_float(r[g * 8 + 5]) * f);
          v.w = pack_bf16(__uint_as_float(r[g * 8 + 6]) * f, __uint_as_float(r[g * 8 + 7]) * f);
          const int chunk = c * 4 + g;
          *reinterpret_cast<uint4*>(stage + (chunk >> 3) * 16384 + sw128_offset(row, chunk & 7)) = v;
        }
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_epi);
    }
    if (tid == 0 && ok && mbar_wait(&bar_epi, 0, abort_w, 33)) {
      tma_store_tile(&mapDV, out_dv, kb * kTile, 0, h, b);
      tma_store_tile(&mapDK, out_dk, kb * kTile, 0, h, b);
      tma_store_commit();
      tma_store_wait_read0();  // of this CTA's shared memory
    }
    BTRACE_ACC(6);
    if ((tid & 127) == 0) BTRACE_ACC_DUMP();
  } else {
    // ------------------------------------------------------------------ dQ reduction warps 8-11, thread = query row
    if (D == 64) reg_inc<136>(); else reg_inc<168>();
    const int w = warp & 3;
    // Each warp owns a stretch of the dQ tile and two private 4 KB boxes in shared memory.  The rows leave in rounds of 32
    // head dimensions: store a round into one box, hand it to a bulk reduce-add, and store the next round into the other
    // box while the first is read.  Nothing else in the CTA waits for these reads.  The accumulator is laid out
    // [tile][query / 32][d / 4][query % 32][d % 4]: a thread stores four head dimensions of its query in 16 bytes without
    // bank conflicts, and a round is 4 KB in one piece there as well as here.  Straight from the registers, as 16-byte
    // reductions of 512 consecutive bytes a warp, the whole backward was 7 to 10 % slower.
    const uint32_t tDQr = tDQ + (static_cast<uint32_t>(w * 32) << 16);
    uint8_t* my_stage = sStage + w * 8192;
    float* acc = p.dq_acc + ((size_t)b * p.H + h) * p.Tp * D;  // + sub * kStretch * D: T <= 2^20 rows of D <= 128, so an int holds it
    for (int i = 0; i < n; ++i) {
      if (!mbar_wait_warp(&bar_ds, i & 1, abort_w, 42)) break;  // from the warps that read the stretch numbers behind the producer's barrier
      const int sub = stretch_of(reinterpret_cast<const uint16_t*>(s_tile)[i % Cfg::kTileSlots * kStretches + w], NB);
      if (!mbar_wait_warp(&bar_g, i & 1, abort_w, 41)) break;
      tc_fence_after();
      if (tid == 2 * kTile) TRACE(1, i, 4);
      uint32_t r[D / 64][64];
#pragma unroll
      for (int c = 0; c < D / 64; ++c) tmem_ld64(tDQr + 64 * c, r[c]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_dqr);  // the dQ columns may be overwritten once all four warps have arrived
      if (tid == 2 * kTile) TRACE(1, i, 5);
      if (sub == kStretches * NB) continue;
      float* dst = acc + sub * (kStretch * D);
#pragma unroll
      for (int k = 0; k < D / 32; ++k) {
        uint8_t* buf = my_stage + (k & 1) * 4096;
        // the box was last used two rounds ago: at most the previous round may still be reading
        if (lane == 0) tma_store_wait_read1();
        __syncwarp();
        const uint32_t* v = &r[k >> 1][32 * (k & 1)];
#pragma unroll
        for (int g = 0; g < 8; ++g)
          *reinterpret_cast<uint4*>(buf + g * 512 + lane * 16) = make_uint4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {
          bulk_reduce_add_f32(dst + k * 1024, buf, 4096);
          tma_store_commit();
        }
      }
      if (tid == 2 * kTile) TRACE(1, i, 6);
    }
    if (lane == 0) tma_store_wait_read0();
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_ptr != 0) {
    if (tid == 0) atomicCAS(P.status, 0, 2000 + *abort_ptr);
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  if (warp == 13) tmem_dealloc(tmem, 512);
}

// The negated statistics -delta and -lse2 per (b, h, t), and zeros for the dQ accumulator.  Rows t >= T of the padded
// arrays get -lse2 = -inf (P = 0) and delta = 0.  HBM-bound, 8 D bytes a row: D / 8 lanes share a row (16 bytes each of
// out and dout), every lane has four rows in flight and writes its 32 bytes of each row's zeros.  A warp per row with
// 4- or 8-byte loads ran at a third of the copy rate, and the memset was a launch of its own (59 + 23 us at 262144 rows of
// D = 128).
template <int D>
__global__ void __launch_bounds__(256) bwd_prep_kernel(const __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ dout,
                                                       const float* __restrict__ lse, int64_t o_sb, int64_t o_sh, int64_t o_st, int64_t d_sb,
                                                       int64_t d_sh, int64_t d_st, int H, int T, int Tp, float* __restrict__ stats,
                                                       float* __restrict__ dq_acc, bool early) {
  constexpr int kLanes = D / 8, kRows = 256 / kLanes, kEach = kTile / kRows < 4 ? kTile / kRows : 4;  // a block covers kRows * kEach rows of one (b, h)
  const int per_bh = Tp / (kRows * kEach);
  wait_previous();
  if (early) let_next_start();
  out = settled(out); dout = settled(dout); lse = settled(lse);
  const int bh = blockIdx.x / per_bh, t0 = (blockIdx.x - bh * per_bh) * (kRows * kEach);
  const int b = bh / H, h = bh - b * H;
  const int r = threadIdx.x / kLanes, c = threadIdx.x % kLanes;
  uint4 ov[kEach], dv[kEach];
#pragma unroll
  for (int i = 0; i < kEach; ++i) {
    const int t = t0 + i * kRows + r;
    ov[i] = dv[i] = make_uint4(0u, 0u, 0u, 0u);
    if (t < T) {
      ov[i] = __ldg(reinterpret_cast<const uint4*>(out + b * o_sb + h * o_sh + (int64_t)t * o_st) + c);
      dv[i] = __ldg(reinterpret_cast<const uint4*>(dout + b * d_sb + h * d_sh + (int64_t)t * d_st) + c);
    }
  }
#pragma unroll
  for (int i = 0; i < kEach; ++i) {
    const int t = t0 + i * kRows + r;
    const int64_t row = (int64_t)bh * Tp + t;
    float4* z = reinterpret_cast<float4*>(dq_acc + row * D);
    z[c] = make_float4(0.f, 0.f, 0.f, 0.f);
    z[c + kLanes] = make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t ow[4] = {ov[i].x, ov[i].y, ov[i].z, ov[i].w}, dw[4] = {dv[i].x, dv[i].y, dv[i].z, dv[i].w};
    float acc = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      acc = fmaf(__uint_as_float(ow[w] << 16), __uint_as_float(dw[w] << 16), acc);
      acc = fmaf(__uint_as_float(ow[w] & 0xffff0000u), __uint_as_float(dw[w] & 0xffff0000u), acc);
    }
#pragma unroll
    for (int s = kLanes / 2; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
    if (c == 0) {
      const float l = t < T ? lse[(int64_t)bh * T + t] : -CUDART_INF_F;
      float* s = stats + row / kStretch * (2 * kStretch) + row % kStretch;
      s[0] = l == -CUDART_INF_F ? -CUDART_INF_F : -l * 1.4426950408889634f;
      s[kStretch] = -acc;
    }
  }
}

// The dQ accumulator [B,H,Tp/32][d / 4][query % 32][d % 4] (fp32, sums of dS K) -> bf16 dq.  A block takes 32 queries of
// one (b, h): four head dimensions of a query are scaled, turned in shared memory and leave as whole rows.
template <int D>
__global__ void __launch_bounds__(256) dq_convert_kernel(const float4* acc, __nv_bfloat16* __restrict__ dq, int64_t sb, int64_t sh,
                                                         int64_t st, int H, int T, int Tp, float scale) {
  __shared__ __align__(16) __nv_bfloat16 s_row[32][D + 8];
  const int per_bh = Tp / 32;
  const int bh = blockIdx.x / per_bh, t0 = (blockIdx.x - bh * per_bh) * 32;
  const float4* src = acc + (size_t)blockIdx.x * (8 * D);
  float4 v[D / 32];
  wait_previous();
#pragma unroll
  for (int i = 0; i < D / 32; ++i) v[i] = ld_v4_here(src + i * 256 + threadIdx.x);
#pragma unroll
  for (int i = 0; i < D / 32; ++i)
    *reinterpret_cast<uint2*>(&s_row[threadIdx.x % 32][(i * 8 + threadIdx.x / 32) * 4]) =
        make_uint2(pack_bf16(v[i].x * scale, v[i].y * scale), pack_bf16(v[i].z * scale, v[i].w * scale));
  __syncthreads();
  const int h = bh % H, b = bh / H;
#pragma unroll
  for (int i = 0; i < D / 64; ++i) {
    const int e = threadIdx.x + i * 256, r = e / (D / 8), c = e % (D / 8);
    if (t0 + r < T) *reinterpret_cast<uint4*>(dq + b * sb + h * sh + (int64_t)(t0 + r) * st + c * 8) = *reinterpret_cast<const uint4*>(&s_row[r][c * 8]);
  }
}

size_t bwd_workspace_bytes(int B, int H, int T, int D) {
  const size_t Tp = (size_t)((T + kTile - 1) / kTile) * kTile;
  const size_t rows = (size_t)B * H * Tp;
  return plan_align(rows * 4) * 2 + plan_align(rows * D * 4);
}

template <int D>
static int launch_bwd_t(const void* q, const void* k, const void* v, const void* out, const void* dout, const float* lse,
                        const int64_t* sq, const int64_t* sk, const int64_t* sv, const int64_t* so, const int64_t* sdo, int B,
                        int H, int T, float scale, PlanView P, MaskArgs M, void* dq, void* dk, void* dv, const int64_t* sdq,
                        const int64_t* sdk, const int64_t* sdv, void* workspace, cudaStream_t stream) {
  const int Tp = P.NB * kTile;
  const size_t rows = (size_t)B * H * Tp;
  char* ws = static_cast<char*>(workspace);
  float* stats = reinterpret_cast<float*>(ws);
  float* dq_acc = reinterpret_cast<float*>(ws + 2 * plan_align(rows * 4));
  CUtensorMap mq, mk, mv, mdo, mqs, mdos, mdk, mdv;
  int r;
  if ((r = cached_tile_map(&mq, q, B, H, T, D, sq[0], sq[1], sq[2], kTile, D))) return r;
  if ((r = cached_tile_map(&mk, k, B, H, T, D, sk[0], sk[1], sk[2], kTile, D))) return r;
  if ((r = cached_tile_map(&mv, v, B, H, T, D, sv[0], sv[1], sv[2], kTile, D))) return r;
  if ((r = cached_tile_map(&mdo, dout, B, H, T, D, sdo[0], sdo[1], sdo[2], kTile, D))) return r;
  if ((r = cached_tile_map(&mqs, q, B, H, T, D, sq[0], sq[1], sq[2], kStretch, 64))) return r;
  if ((r = cached_tile_map(&mdos, dout, B, H, T, D, sdo[0], sdo[1], sdo[2], kStretch, 64))) return r;
  if ((r = cached_tile_map(&mdk, dk, B, H, T, D, sdk[0], sdk[1], sdk[2], kTile, D))) return r;
  if ((r = cached_tile_map(&mdv, dv, B, H, T, D, sdv[0], sdv[1], sdv[2], kTile, D))) return r;
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return -120;
  if (!attr_done[dev]) {
    if (cudaFuncSetAttribute(attn_bwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdSmem<D>::kBytes) != cudaSuccess)
      return -120;
    attr_done[dev] = true;
  }
  constexpr int kPrepRows = 256 / (D / 8) * (kTile / (256 / (D / 8)) < 4 ? kTile / (256 / (D / 8)) : 4);
  BwdParams p;
  p.plan = P; p.mask = M; p.stats = stats; p.dq_acc = dq_acc;
  p.dk = static_cast<__nv_bfloat16*>(dk); p.dv = static_cast<__nv_bfloat16*>(dv);
  for (int i = 0; i < 3; ++i) { p.dk_s[i] = sdk[i]; p.dv_s[i] = sdv[i]; }
  p.H = H; p.Tp = Tp; p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  {  // heads per group: their Q and dO (2 x T x D bf16 each) stay within TS2TS_BWD_GROUP_MB, a quarter of the L2
    const long long qdo_bytes = 4ll * T * D;
    long long g = (static_cast<long long>(TS2TS_BWD_GROUP_MB) << 20) / (qdo_bytes > 0 ? qdo_bytes : 1);
    p.head_group = (int)(g < 1 ? 1 : (g > H ? H : g));
  }
  BTRACE_ATTACH(p, stream);
  // The main kernel's blocks set themselves up and bring in K and V under the preparation where the launches are short.  us, one after the other -> overlapping: linked 1024,
  // H = 4, D = 64 22.4 -> 21.1; causal 1024, H = 4, D = 128 28.2 -> 26.7.  Between one tile an SM and the line it goes either way by 1 to 4 % (D = 128, documents 2 x 2600, H = 8
  // 59.8 -> 57.4, linked 4096, H = 7 83.0 -> 86.9); beyond 384 tiles at D = 128 and 768 at D = 64 launches lose (linked 8k, H = 12, D = 64, 768 tiles 91.5 -> 93.6).
  // The conversion does not start under the main kernel: a trigger there costs more than it gives (linked 5003, H = 12, D = 64 62.5 -> 63.6, 16k, H = 16, D = 128 961 -> 982).
  const bool early = (long long)B * H * P.NB * D <= 384 * 128;
  cudaError_t launched = launch_after(bwd_prep_kernel<D>, dim3((unsigned)(rows / kPrepRows)), 256, 0, stream, static_cast<const __nv_bfloat16*>(out),
                                      static_cast<const __nv_bfloat16*>(dout), lse, so[0], so[1], so[2], sdo[0], sdo[1], sdo[2], H, T, Tp, stats, dq_acc, early);
  if (launched == cudaSuccess) {
    ProfileScope timed(1, stream);
    launched = launch_after(attn_bwd_kernel<D>, dim3((unsigned)B * H * P.NB), kBwdThreads, BwdSmem<D>::kBytes, stream, mq, mk, mv, mdo, mqs, mdos, mdk, mdv, p);
  }
  if (launched == cudaSuccess)
    launched = launch_after(dq_convert_kernel<D>, dim3((unsigned)(rows / 32)), 256, 0, stream, reinterpret_cast<const float4*>(dq_acc),
                            static_cast<__nv_bfloat16*>(dq), sdq[0], sdq[1], sdq[2], H, T, Tp, scale);
  BTRACE_DUMP(stream);
  const cudaError_t last = cudaGetLastError();
  return launched == cudaSuccess && last == cudaSuccess ? 0 : -121;
}

int launch_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout, const float* lse, const int64_t* sq,
               const int64_t* sk, const int64_t* sv, const int64_t* so, const int64_t* sdo, int B, int H, int T, int D, float scale,
               PlanView P, MaskArgs M, void* dq, void* dk, void* dv, const int64_t* sdq, const int64_t* sdk, const int64_t* sdv,
               void* workspace, cudaStream_t stream) {
  if (D == 128)
    return launch_bwd_t<128>(q, k, v, out, dout, lse, sq, sk, sv, so, sdo, B, H, T, scale, P, M, dq, dk, dv, sdq, sdk, sdv, workspace, stream);
  if (D == 64)
    return launch_bwd_t<64>(q, k, v, out, dout, lse, sq, sk, sv, so, sdo, B, H, T, scale, P, M, dq, dk, dv, sdq, sdk, sdv, workspace, stream);
  return -122;
}

// --------------------------------------------------------------------------------------------------------------
// Scratch that lives inside the library, for ts2ts_attn_bwd_noalloc (see include/ts2ts_attn.h).
//
// `g_static_scratch` is a device array.  Host code must not use the name as a pointer: on the host it is only a
// handle, and a kernel handed that handle would read or write unrelated memory.  The device address is asked for
// once per device with cudaGetSymbolAddress, with that device current, and cached.
constexpr size_t kStaticScratchBytes = size_t(64) << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

int bwd_static_scratch(void** ptr, size_t* bytes) {
  static void* cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -130;
  if (cached[dev] == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || p == nullptr) return -131;
    cached[dev] = p;
  }
  *ptr = cached[dev];
  *bytes = kStaticScratchBytes;
  return 0;
}

}  // namespace ts2ts
