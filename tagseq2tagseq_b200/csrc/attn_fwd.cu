// Masked flash-attention forward for sm_100a.
//
// Persistent kernel, one CTA per SM.  A work item is a pair of adjacent 128-row query tiles (2p, 2p+1) of one
// (batch, head); a CTA's first item is its own number, further ones are drawn from a ticket counter, group of heads after group of heads, inside a group the pairs with the
// most key tiles first, so the tiles that run at the same time share K/V in L2 and the long items start early.  Each query tile of the pair belongs to a "team":
//   softmax team t   4 warps, one thread per query row (setmaxnreg 216)
//   issuer t         1 thread issuing the team's tcgen05.mma
// and one producer thread feeds both teams with TMA.  Both teams walk the same ascending stream of key tiles (the
// union of their two lists; a team simply does nothing for a tile only the other one reads), so every K/V tile is
// brought into shared memory once per pair.  Per key tile and team:
//   tcgen05   S = Q K^T                       (bf16 x bf16 -> fp32, 128 columns of tensor memory)
//   softmax   the row's 128 scores are read into registers in one go and the S columns are handed back at
//             once, so that the issuer can compute S of the NEXT key tile while this one is being exponentiated;
//             mask (partial tiles only: one select per element against a per-row 128-bit column mask that the pre-pass
//             worked out; 32-column chunks that are masked for a whole warp are skipped), online softmax in
//             base 2, P -> bf16 -> tensor memory (D = 64) or shared memory (D = 128; K-major, 128-byte swizzle)
//   tcgen05   O += P V                        (V MN-major; with P in tensor memory the first 64 keys as soon as theirs is there)
// P needs a place other than the scores it is made from, or S of the next tile could not be computed meanwhile.  At D = 64
// tensor memory has room for it (S0 | S1 | O0 | O1 | P0 | P1), which takes 128 KB a pair of tiles out of the shared-memory
// pipe that the MMA operands fill (H = 16, causal 4k batch 4: 239 -> 222 us, linked 16k: 370 -> 348).  At D = 128 it has not: with P
// over its own scores a team waited 1570 clocks a tile for S where it waits 240 (causal 4k); with P in tensor memory and one score buffer
// for both teams causal 4k batch 4 took 296 us instead of 304, but linked 16k 406 instead of 390 and two linked 32k packs 4160 instead of
// 4125, because teams whose tiles differ then wait for each other's reads.
// The accumulator is rescaled lazily: only when a row's running maximum grows by more than 2^8.
// K/V tiles travel through one ring of shared-memory slots in the order K0, K1, V0, K2, V1, ... (K runs one tile
// ahead of V because S is computed one tile ahead of P V).  Launches that are as long as their longest list have the teams share a query tile
// instead (launch_fwd_t): the tiles of its list go to them in turn, K two tiles ahead of V so that either team's S is computed ahead there too
// (us with K one tile ahead -> two: causal 4096, H = 8, D = 128 51 -> 45, linked 16k, H = 2, D = 64 75 -> 66, linked 1024, H = 4 18.5 -> 16.6),
// and team 0 adds up both parts at the end, straight from tensor memory.  At the end of an item each softmax thread reads its
// row of O out of tensor memory and frees it for the next item; the normalised rows leave through shared memory and TMA stores, a
// warp's 32 rows at a time, while the issuers already work on the next item.
//
// Shared memory at D = 128: Q0 Q1 (64 KB), P0 P1 (64 KB), three K/V slots (96 KB); at D = 64: Q0 Q1 (32 KB), O0 O1 (32 KB),
// eight slots (128 KB).
//
// Computes what the reference obtains from PyTorch FlexAttention's forward
// (model/modules/layer.py:33 via tunalab FlexSelfAttention; semantics in
// torch/_higher_order_ops/flex_attention.py:218-287): O = softmax(scale QK^T +
// mask) V, LSE in natural log, a fully masked row gives O = 0 and LSE = -inf.
#include "launch.cuh"
#include "plan.h"
#include "profile.h"
#include "ptx.cuh"
#include "tma_host.h"

#include <limits.h>
#include <math_constants.h>

#include <type_traits>

// A debug build may name a private header that defines the three hooks below to record clock64() stamps.
#ifdef TS2TS_TRACE_HEADER
#include TS2TS_TRACE_HEADER
#else
#define TS2TS_TRACE_FIELDS
#define FTRACE(role, step, ev) do { } while (0)
#define FTRACE_SPAN(which) do { } while (0)
#define FTRACE_CTA(slot, value) do { } while (0)
#define FTRACE_ACC_DECL
#define FTRACE_ACC(k) do { } while (0)
#define FTRACE_ACC_DUMP(team) do { } while (0)
#define FTRACE_ATTACH(params, stream) do { } while (0)
#define FTRACE_DUMP(stream) do { } while (0)
#endif

#ifndef TS2TS_FWD_GROUP_MB
// K/V bytes of the heads whose work items are interleaved in the ticket order.  Measured on the 32k masks: 136 MB
// (8 heads) is 5-7 % faster than 64 MB on the two sparser masks, equal on the densest, 2 % slower on plain causal.
#define TS2TS_FWD_GROUP_MB 136
#endif
#ifndef TS2TS_FWD_FOLD_MB
// K/V bytes of the whole batch (in 2^20) up to which its elements are ordered as one: the first ranks of all of them come before any second
// one, so that every element's heavy items start early.  A little under the L2's 126e6 bytes.  us, one after the other -> as one, D = 64 unless
// noted: causal 4 x 2039, H = 8 56.3 -> 42.7; linked 4 x 14724, H = 3 248 -> 223; D = 128: documents 4 x 3269, H = 8 51.1 -> 47.2; linked 4 x 4096, H = 12
// (96) 197 -> 172, H = 14 (112) 169 -> 145; linked 2 x 16384, H = 6 (96) 323 -> 294.  Even elements gain little or nothing: causal 4 x 4096, H = 13 (104)
// 245 -> 243, 2 x 8192, H = 10 to 14 (80 to 112) +- 1-2 %, linked 2 x 14336, H = 10 to 14, D = 64 (70 to 98) -1 to +1 %.  Beyond the line: linked 4 x 4096, H = 15 (120)
// 185 -> 162, but causal 4 x 4096, H = 16 (128) 293 -> 308.  The backward gains nothing from it (its blocks are many).
#define TS2TS_FWD_FOLD_MB 112
#endif

namespace ts2ts {

struct FwdParams {
  PlanView plan;
  MaskArgs mask;
  float* lse;            // [B,H,T]
  __nv_bfloat16* out;
  int64_t o_sb, o_sh, o_st;
  int H;
  int n_pairs, n_tiles;  // B * H * ceil(NB / 2) and B * H * NB: the work items as pairs and as shared query tiles
  int heads;             // heads of a stretch of the ticket order: H, or B * H where the batch elements are one
  int head_group;        // heads whose items are interleaved in the ticket order
  float scale_log2;      // softmax scale * log2(e)
  TS2TS_TRACE_FIELDS
};

constexpr int kFwdThreads = 384;   // warps 0-3 softmax team 0, 4-7 team 1, 8-9 MMA issuers, 10 TMA producer, 11 idle
constexpr int kFwdIssuerWarp = 8;  // + team
constexpr int kFwdProducerWarp = 10;
constexpr int kFwdItemSlots = 2;
constexpr uint32_t kNoMasks = 0xffffffffu;
template <uint32_t N> __device__ __forceinline__ void fwd_reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <uint32_t N> __device__ __forceinline__ void fwd_reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
constexpr float kRescaleThreshold = 8.0f;
// A wait that is not asked how it ended.  Only its first poll is inline: with the loops inside the tile's code, and no exit from
// them, full tiles took 2 % longer (causal 4k batch 4, D = 64: 226 instead of 220 us).
__device__ __noinline__ void wait_longer(uint64_t* bar, uint32_t parity, volatile int* abort_word, int code) {
  mbar_wait(bar, parity, abort_word, code);
}

template <int D>
struct FwdSmem {
  static constexpr int kSub = D / 64;
  static constexpr int kTileBytes = kTile * D * 2;
  static constexpr bool kTmemP = D == 64;                    // P in tensor memory
  static constexpr int kPBytes = kTile * D * 2;              // at D = 128 P's place; output rows always leave through it
  static constexpr int kStages = D == 128 ? 3 : 8;
  static constexpr int kQ = 0;                               // two Q tiles
  static constexpr int kP = 2 * kTileBytes;                  // two P (or O) tiles
  static constexpr int kRing = kP + 2 * kPBytes;             // K/V slots
  static constexpr int kSmall = kRing + kStages * kTileBytes;
  static constexpr int kBars = 21 + 2 * kStages;
  static constexpr int kSmallBytes = kTile * 8 + kFwdItemSlots * (48 + 32 * (kMaskRuns + 1)) + kBars * 8 + 8 + 4 * kStages;  // row statistics, items, barriers, words
  static constexpr int kBytes = kSmall + kSmallBytes + 1024;  // + alignment slack
  // tensor-memory columns of team t
  static __host__ __device__ constexpr int score_col(int t) { return t * kTile; }
  static __host__ __device__ constexpr int out_col(int t) { return 2 * kTile + t * D; }
  static __host__ __device__ constexpr int p_col(int t) { return 2 * kTile + 2 * D + t * 64; }  // kTmemP
};

// One work item as the producer publishes it in shared memory, with all that a softmax warp would otherwise fetch from global memory, four accesses one after
// the other, before its first tile (with the numbers of heads and rows read back from here at the end instead of kept, us: causal 4k batch 4, H = 16, D = 64
// 222 -> 213, D = 128 298 -> 282, linked 16k, H = 12, D = 64 256 -> 252).  Teams that share a query tile take every other entry of its list.
struct alignas(16) FwdItem {
  int code, b, h, qb;           // code < 0: no more work; the first team's query tile (the second one's is the next, or the same where they share it)
  int n[2], n_runs[2];          // key tiles and runs of each team's query tile
  int first[2][2];              // the first two list entries of each team
  Run runs[2][kMaskRuns + 1];   // the first runs of each team's query tile (of the shared one: [0])
};
static_assert(sizeof(FwdItem) == 48 + 2 * 16 * (kMaskRuns + 1), "");
// Ticket order: batch elements one after the other, or, in short launches, as one (`heads` = B * H); inside one, groups of G heads;
// inside a group all heads' heaviest items first, then their second heaviest, and so on.  The group bounds the K/V working set that has
// to stay in L2, and the long items of the last group still start well before the end of the launch.
// Returns where the plan says which query tile (or pair of them) it is.
__device__ __forceinline__ const int32_t* item_place(const PlanView& P, int H, int heads, int G, bool split, int code, int& b, int& h) {
  const int NI = split ? P.NB : (P.NB + 1) / 2;
  const int per_b = heads * NI;
  const int b0 = code / per_b;
  const int r1 = code - b0 * per_b;
  const int g = r1 / (G * NI);
  const int r2 = r1 - g * G * NI;
  const int gsize = min(G, heads - g * G);
  const int rank = r2 / gsize;
  h = g * G + (r2 - rank * gsize);
  const int more = h / H;  // batch elements past b0
  b = b0 + more;
  h -= more * H;
  return (split ? P.fwd_order : P.pair_order) + (size_t)b * NI + rank;
}
// The rest of the item, one round of loads.
__device__ __forceinline__ void read_item(const PlanView& P, bool split, int at, FwdItem& it) {
  at = min(max(at, 0), (split ? P.NB : (P.NB + 1) / 2) - 1);
  it.qb = split ? at : 2 * at;
  const bool two = !split && it.qb + 1 < P.NB;
  const size_t row0 = (size_t)it.b * P.NB + it.qb, row1 = two ? row0 + 1 : row0;
  const int32_t *l0 = P.fwd_idx + row0 * P.NB, *l1 = P.fwd_idx + row1 * P.NB;
  const int c0 = ld_nc_i32_here(&P.fwd_cnt[row0]), c1 = ld_nc_i32_here(&P.fwd_cnt[row1]);
  const int r0 = ld_nc_i32_here(&P.run_cnt[row0]), r1 = ld_nc_i32_here(&P.run_cnt[row1]);
  // entries past a list's end are there up to its NB-th and are not looked at
  const int e00 = ld_nc_i32_here(l0), e01 = ld_nc_i32_here(l0 + min(split ? 2 : 1, P.NB - 1));
  const int e10 = ld_nc_i32_here(l1 + (split ? min(1, P.NB - 1) : 0)), e11 = ld_nc_i32_here(l1 + min(split ? 3 : 1, P.NB - 1));
  const int n0 = min(max(c0, 0), P.NB);
  it.n[0] = split ? (n0 + 1) / 2 : n0;
  it.n[1] = split ? n0 / 2 : two ? min(max(c1, 0), P.NB) : 0;
  it.n_runs[0] = r0; it.n_runs[1] = r1;
  it.first[0][0] = e00; it.first[0][1] = e01; it.first[1][0] = e10; it.first[1][1] = e11;
}
// What a ring slot holds, written by the producer next to the slot.
enum : uint32_t {
  kRingTeam0 = 1u, kRingTeam1 = 2u,     // the tile is on the list of team 0 / 1
  kRingIsV = 4u,                        // V tile (else K)
  kRingFirst0 = 8u, kRingFirst1 = 16u,  // the team's first tile of the item
  kRingLast0 = 32u, kRingLast1 = 64u,   // the team's last tile of the item
  kRingEnd = 128u,                      // no more work
};
// The key tiles of an item in the order of the ring: the ascending merge of the teams' lists, or the one list of teams that share a
// query tile, whose tiles go to the teams in turn.  next() returns the next key tile, -1 at the end, and
// -2 when an entry is not a tile number (the plan does not belong to this call); `info` gets the kRing* bits.
struct UnionWalk {
  const int32_t *l0, *l1;
  int n0, n1, i0, i1, NB;
  bool split;
  __device__ __forceinline__ void start(const PlanView& P, const FwdItem& it, bool shared) {
    l0 = P.fwd_idx + ((size_t)it.b * P.NB + it.qb) * P.NB;
    l1 = shared ? l0 : l0 + P.NB;
    n0 = it.n[0]; n1 = it.n[1]; i0 = i1 = 0; NB = P.NB; split = shared;
  }
  __device__ __forceinline__ int next(uint32_t& info) {
    if (split) {
      const int n = n0 + n1;
      if (i0 >= n) return -1;
      const int kb = static_cast<int>(__ldg(l0 + i0) & ~kFullBit);
      if (kb < 0 || kb >= NB) return -2;
      info = (kRingTeam0 | (i0 < 2 ? kRingFirst0 : 0u) | (i0 >= n - 2 ? kRingLast0 : 0u)) << (i0 & 1);
      ++i0;
      return kb;
    }
    const int a = i0 < n0 ? static_cast<int>(__ldg(l0 + i0) & ~kFullBit) : INT_MAX;
    const int c = i1 < n1 ? static_cast<int>(__ldg(l1 + i1) & ~kFullBit) : INT_MAX;
    const int kb = min(a, c);
    if (kb == INT_MAX) return -1;
    if (kb < 0 || kb >= NB) return -2;
    info = 0;
    if (a == kb) {
      info |= kRingTeam0 | (i0 == 0 ? kRingFirst0 : 0u) | (i0 == n0 - 1 ? kRingLast0 : 0u);
      ++i0;
    }
    if (c == kb) {
      info |= kRingTeam1 | (i1 == 0 ? kRingFirst1 : 0u) | (i1 == n1 - 1 ? kRingLast1 : 0u);
      ++i1;
    }
    return kb;
  }
};

// 128-bit mask of the key columns of tile kb that row `row` of tile qb may read, before causality, from the run lists: the
// way out for rows that the plan's mask table does not cover.  Kept out of line: it is rare, and the softmax loop's code is
// what the instruction cache has to hold.
__device__ __noinline__ uint4 row_mask(const PlanView& P, const MaskArgs& M, int b, int qb, int kb, int row) {
  const int q = qb * kTile + row;
  if (q >= P.T) return make_uint4(0u, 0u, 0u, 0u);
  const int mydoc = M.doc[(size_t)b * P.T + q], myrow = M.row[(size_t)b * P.T + q];
  const int64_t* link_row = (M.link != nullptr && myrow >= 0 && myrow < M.R) ? M.link + ((size_t)b * M.R + myrow) * M.W : nullptr;
  const size_t tk = (size_t)b * P.NB + kb;
  const int4* runs = reinterpret_cast<const int4*>(P.runs + tk * kTile);
  const int n = min(__ldg(&P.run_cnt[tk]), kTile), n_valid = min(kTile, P.T - kb * kTile);
  uint32_t bits[4] = {0u, 0u, 0u, 0u};
  int4 cur = __ldg(runs);
  uint32_t lo[4];
  prefix_mask(cur.x, lo);
  for (int r = 0; r < n; ++r) {
    const int4 nx = r + 1 < n ? __ldg(runs + r + 1) : make_int4(n_valid, 0, 0, 0);
    uint32_t hi[4];
    prefix_mask(nx.x, hi);
    bool allowed = cur.y == mydoc;
    if (!allowed && link_row != nullptr && cur.w >= 0 && cur.w < 64 * M.W)
      allowed = (static_cast<unsigned long long>(__ldg(link_row + (cur.w >> 6))) >> (cur.w & 63)) & 1ull;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      if (allowed) bits[w] |= hi[w] & ~lo[w];
      lo[w] = hi[w];
    }
    cur = nx;
  }
  return make_uint4(bits[0], bits[1], bits[2], bits[3]);
}

// The last CTA to leave puts the ticket counter back to zero for the next launch.
__device__ __forceinline__ void fwd_leave(const PlanView& P) {
  __threadfence();
  const int done = atomicAdd(&P.status[kFwdDone], 1);
  if (done == static_cast<int>(gridDim.x) - 1) {
    P.status[kFwdTicket] = 0;
    P.status[kFwdDone] = 0;
    __threadfence();
  }
}

// Where the pieces of a CTA's shared memory lie.
template <int D>
struct FwdPlaces {
  using Cfg = FwdSmem<D>;
  uint8_t *raw, *smem;
  uint8_t* sQ;
  uint8_t* sP;
  uint8_t* sRing;
  float2* s_merge;  // [row] maximum and sum of team 1
  FwdItem* s_item;  // [2]
  uint64_t* bars;
  uint64_t* bar_item_full;  // [2] the producer published an item
  uint64_t* bar_item_empty;  // [2] the eight softmax warps are through with it
  uint64_t* bar_q_full;  // [team] Q tile landed
  uint64_t* bar_q_free;  // [team] last S of the item complete: the Q buffer may be reloaded
  uint64_t* bar_s;  // [team] S of the tile is in tensor memory
  uint64_t* bar_sfree;  // [team] S read into registers: its columns may be overwritten
  uint64_t* bar_p;  // [team] P of the tile (D = 64: of its last 64 keys) is written
  uint64_t* bar_pv;  // [team] P V of the tile complete: P free, O consistent
  uint64_t* bar_ofree;  // [team] O of the item read out of tensor memory
  uint64_t* bar_p0;  // [team] P of the tile's first 64 keys is in tensor memory and O is rescaled (D = 64)
  uint64_t* bar_merge;  // team 1's part of a shared query tile is in tensor memory, its row statistics in s_merge
  uint64_t* bar_ring_full;  // [kStages] K or V tile landed in the slot
  uint64_t* bar_ring_free;  // [kStages] both issuers are done with the slot
  uint32_t* tmem_slot;
  int* abort_w;
  uint32_t* s_ring_info;  // [kStages] kRing* bits of what each slot holds
  __device__ __forceinline__ explicit FwdPlaces(uint8_t* base) : raw(base) {
    // Plain pointer arithmetic (no round trip through an integer) keeps the shared address space visible to the
    // compiler, so every access becomes a shared-memory instruction instead of a generic one.
    smem = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
    sQ = smem + Cfg::kQ;
    sP = smem + Cfg::kP;
    sRing = smem + Cfg::kRing;
    s_merge = reinterpret_cast<float2*>(smem + Cfg::kSmall);
    s_item = reinterpret_cast<FwdItem*>(s_merge + kTile);
    bars = reinterpret_cast<uint64_t*>(s_item + kFwdItemSlots);
    bar_item_full = bars;
    bar_item_empty = bars + 2;
    bar_q_full = bars + 4;
    bar_q_free = bars + 6;
    bar_s = bars + 8;
    bar_sfree = bars + 10;
    bar_p = bars + 12;
    bar_pv = bars + 14;
    bar_ofree = bars + 16;
    bar_p0 = bars + 18;
    bar_merge = bars + 20;
    bar_ring_full = bars + 21;
    bar_ring_free = bars + 21 + Cfg::kStages;
    tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::kBars);
    abort_w = reinterpret_cast<int*>(tmem_slot + 1);
    s_ring_info = tmem_slot + 2;
  }
};

// Barriers and tensor memory; nothing here looks at memory that an earlier launch may have written.  Returns the tensor memory's address.
template <int D>
__device__ __forceinline__ uint32_t fwd_setup(const FwdPlaces<D>& at) {
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    *at.abort_w = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(&at.bar_item_full[i], 1);
      mbar_init(&at.bar_item_empty[i], 8);
      mbar_init(&at.bar_q_full[i], 1);
      mbar_init(&at.bar_q_free[i], 1);
      mbar_init(&at.bar_s[i], 1);
      mbar_init(&at.bar_sfree[i], 4);  // one arrival per softmax warp
      mbar_init(&at.bar_p[i], 4);
      mbar_init(&at.bar_p0[i], 4);
      mbar_init(&at.bar_pv[i], 1);
      mbar_init(&at.bar_ofree[i], 4);
    }
    mbar_init(at.bar_merge, 4);
    for (int i = 0; i < FwdSmem<D>::kStages; ++i) {
      mbar_init(&at.bar_ring_full[i], 1);
      mbar_init(&at.bar_ring_free[i], 2);
    }
    fence_mbar_init();
  }
  __syncthreads();
  if (warp == kFwdIssuerWarp) {
    tmem_alloc(at.tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return *at.tmem_slot;
}

// kShared: the two teams of a CTA share a query tile and take its key tiles in turn, instead of a query tile of a pair each.
// `first_at`: for the producer, what the plan says about the CTA's first item.
template <int D, bool kShared>
__device__ __forceinline__ void fwd_items(const CUtensorMap& mapQ, const CUtensorMap& mapK, const CUtensorMap& mapV, const CUtensorMap& mapO, const FwdParams& p,
                                          const FwdPlaces<D>& at, uint32_t tmem, int first_at) {
  using Cfg = FwdSmem<D>;
  constexpr int kStages = Cfg::kStages;
  uint8_t* const sQ = at.sQ;
  uint8_t* const sP = at.sP;
  uint8_t* const sRing = at.sRing;
  float2* const s_merge = at.s_merge;
  FwdItem* const s_item = at.s_item;
  uint64_t* const bars = at.bars;
  uint64_t* const bar_item_full = at.bar_item_full;
  uint64_t* const bar_item_empty = at.bar_item_empty;
  uint64_t* const bar_q_full = at.bar_q_full;
  uint64_t* const bar_q_free = at.bar_q_free;
  uint64_t* const bar_s = at.bar_s;
  uint64_t* const bar_sfree = at.bar_sfree;
  uint64_t* const bar_p = at.bar_p;
  uint64_t* const bar_pv = at.bar_pv;
  uint64_t* const bar_ofree = at.bar_ofree;
  uint64_t* const bar_p0 = at.bar_p0;
  uint64_t* const bar_merge = at.bar_merge;
  uint64_t* const bar_ring_full = at.bar_ring_full;
  uint64_t* const bar_ring_free = at.bar_ring_free;
  uint32_t* const tmem_slot = at.tmem_slot;
  int* const abort_w = at.abort_w;
  uint32_t* const s_ring_info = at.s_ring_info;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const PlanView& P = p.plan;
  const int NB = P.NB;
  const int n_items = kShared ? p.n_tiles : p.n_pairs;
  volatile int* abort_v = abort_w;

  if (warp >= 8) {
    fwd_reg_dec<72>();  // register pool: 256 x 216 + 128 x 72 = 384 x 168
    if (warp == kFwdProducerWarp && lane == 0) {
      // ------------------------------------------------------------------ TMA producer
      // Walks the key-tile lists (the only role that reads them from global memory besides the softmax threads) and
      // tells the issuers through a word per ring slot what the slot holds and which team uses it.
      tma_prefetch_desc(&mapQ); tma_prefetch_desc(&mapK); tma_prefetch_desc(&mapV);
      uint32_t ring = 0;             // ring slots filled so far
      uint32_t q_loads[2] = {0, 0};  // Q tiles loaded so far, per team
      bool ok = true;
      auto fill = [&](const CUtensorMap* map, uint32_t info, int kb, int h, int b) {
        const uint32_t slot = ring % kStages, use = ring / kStages;
        if (use > 0 && !mbar_wait(&bar_ring_free[slot], (use - 1) & 1, abort_v, 11)) return false;
        s_ring_info[slot] = info;
        if (map != nullptr) {
          mbar_expect_tx(&bar_ring_full[slot], Cfg::kTileBytes);
          tma_load_tile(sRing + slot * Cfg::kTileBytes, map, &bar_ring_full[slot], kb * kTile, 0, h, b);
        } else {
          mbar_arrive(&bar_ring_full[slot]);  // end marker: nothing to load
        }
        ++ring;
        return true;
      };
      for (uint32_t it = 0; ok; ++it) {
        const uint32_t is = it % kFwdItemSlots;
        if (it >= kFwdItemSlots && !mbar_wait(&bar_item_empty[is], (it / kFwdItemSlots - 1) & 1, abort_v, 12)) break;
        // The first item of a CTA is its own number; the next one is drawn once all copies of the last have been asked for: earlier draws
        // cost balance (at the start of the last item 8-15 %, linked 16k, H = 12, D = 64).
        int code = it == 0 ? static_cast<int>(blockIdx.x) : static_cast<int>(gridDim.x) + atomicAdd(&P.status[kFwdTicket], 1);
        if (code >= n_items) {
          s_item[is].code = -1;
          mbar_arrive(&bar_item_full[is]);
          fill(nullptr, kRingEnd, 0, 0, 0);
          break;
        }
        FwdItem& item = s_item[is];
        int h, b;
        const int32_t* place = item_place(P, p.H, p.heads, p.head_group, kShared, code, b, h);
        item.code = code; item.b = b; item.h = h;
        read_item(P, kShared, it == 0 ? first_at : ld_nc_i32_here(place), item);
        const int qb = item.qb, n_own[2] = {item.n[0], item.n[1]};
        auto publish = [&]() {
          const int tiles = P.q_mask == nullptr ? 0 : kShared || qb + 1 >= NB ? 1 : 2;
          mbar_expect_tx(&bar_item_full[is], tiles * (int)sizeof(item.runs[0]));
          for (int t = 0; t < tiles; ++t) bulk_load(item.runs[t], P.runs + ((size_t)b * NB + qb + t) * kTile, sizeof(item.runs[0]), &bar_item_full[is]);
        };
        if (it > 0) publish();  // the first time the tiles' copies are the ones to hurry
        for (int t = 0; t < 2 && ok; ++t) {
          if (n_own[t] == 0) continue;
          if (q_loads[t] > 0 && !mbar_wait(&bar_q_free[t], (q_loads[t] - 1) & 1, abort_v, 13)) { ok = false; break; }
          mbar_expect_tx(&bar_q_full[t], Cfg::kTileBytes);
          tma_load_tile(sQ + t * Cfg::kTileBytes, &mapQ, &bar_q_full[t], (kShared ? qb : qb + t) * kTile, 0, h, b);
          ++q_loads[t];
        }
        if (!ok) break;
        UnionWalk w;
        w.start(P, item, kShared);
        // The tiles whose K is in the ring and whose V is not yet: one, or two where the teams share a query tile, so that either team's
        // next K comes ahead of its current V and its next S is computed during the softmax of this one.
        constexpr int kAhead = kShared ? 2 : 1;
        uint32_t infos[kAhead + 1];
        int tiles[kAhead + 1];
        auto next_k = [&](int at) {  // the next tile of the walk into place `at`, its K into the ring
          tiles[at] = w.next(infos[at]);
          if (tiles[at] == -2) { atomicCAS(abort_w, 0, 14); return false; }
          return tiles[at] < 0 || fill(&mapK, infos[at], tiles[at], h, b);
        };
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          tiles[i] = -1;
          if (ok && (i == 0 || tiles[i - 1] >= 0)) ok = next_k(i);
          if (i == 0 && it == 0) publish();
        }
        while (tiles[0] >= 0 && ok) {
          tiles[kAhead] = -1;
          if (tiles[kAhead - 1] >= 0) ok = next_k(kAhead);
          if (ok) ok = fill(&mapV, infos[0] | kRingIsV, tiles[0], h, b);
#pragma unroll
          for (int i = 0; i < kAhead; ++i) {
            tiles[i] = tiles[i + 1];
            infos[i] = infos[i + 1];
          }
        }
      }
    } else if ((warp == kFwdIssuerWarp || warp == kFwdIssuerWarp + 1) && lane == 0) {
      // ------------------------------------------------------------------ MMA issuer of team t
      // Takes the ring slots in order: waits until a slot is filled, uses it if the tile is on this team's list
      // (S = Q K^T for a K slot, O += P V for a V slot) and hands it back.  It reads shared memory only.
      const int t = warp - kFwdIssuerWarp;
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);
      constexpr uint32_t idesc_pv = make_idesc_bf16(128, D, false, true);
      // descriptor halves: K-major operands (Q, K, P) step 32 B inside a 128-byte row and 16 KB between two
      // 64-column halves; the MN-major operand (V) steps 16 key rows = 2048 B
      constexpr uint32_t hi_k = desc_hi(1024);
      const uint32_t q_lo = desc_lo(smem_u32(sQ + t * Cfg::kTileBytes), 16);
      const uint32_t p_lo = desc_lo(smem_u32(sP + t * Cfg::kPBytes), 16);
      const uint32_t k_ring_lo = desc_lo(smem_u32(sRing), 16), v_ring_lo = desc_lo(smem_u32(sRing), 16384);
      const uint32_t tS = tmem + Cfg::score_col(t), tO = tmem + Cfg::out_col(t), tP = tmem + Cfg::p_col(t);
      const uint32_t mine_bit = kRingTeam0 << t, first_bit = kRingFirst0 << t, last_bit = kRingLast0 << t;
      uint32_t n_s = 0;      // S tiles issued by this team so far
      uint32_t n_pv = 0;     // P V tiles issued so far
      uint32_t n_items = 0;  // items this team has started
      for (uint32_t ring = 0;; ++ring) {
        const uint32_t slot = ring % kStages, use = ring / kStages;
        if (!mbar_wait(&bar_ring_full[slot], use & 1, abort_v, 23)) break;
        const uint32_t info = s_ring_info[slot];
        if (info & kRingEnd) break;
        if (!(info & mine_bit)) {
          mbar_arrive(&bar_ring_free[slot]);
          continue;
        }
        if (!(info & kRingIsV)) {
          if ((info & first_bit) && !mbar_wait(&bar_q_full[t], n_items & 1, abort_v, 22)) break;
          if (info & first_bit) ++n_items;
          if (n_s > 0 && !mbar_wait(&bar_sfree[t], (n_s - 1) & 1, abort_v, 24)) break;
          tc_fence_after();
          FTRACE(2 * t, n_s, 0);
          const uint32_t k_lo = k_ring_lo + slot * (Cfg::kTileBytes >> 4);
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
            mma_ss2(tS, q_lo + off, hi_k, k_lo + off, hi_k, idesc_s, kk > 0);
          }
          mma_commit(&bar_s[t]);
          FTRACE(2 * t, n_s, 1);
          ++n_s;
          if (info & last_bit) mma_commit(&bar_q_free[t]);
          mma_commit(&bar_ring_free[slot]);
        } else {
          if (!mbar_wait(Cfg::kTmemP ? &bar_p0[t] : &bar_p[t], n_pv & 1, abort_v, 26)) break;
          // the first P V of an item overwrites O: the previous item's rows must have been read out
          // (n_items counts this item already, so the previous one is n_items - 2)
          if ((info & first_bit) && n_items > 1 && !mbar_wait(&bar_ofree[t], (n_items - 2) & 1, abort_v, 27)) break;
          tc_fence_after();
          FTRACE(2 * t, n_pv, 2);
          const uint32_t v_lo = v_ring_lo + slot * (Cfg::kTileBytes >> 4);
          const uint32_t acc0 = (info & first_bit) ? 0u : 1u;
          if constexpr (Cfg::kTmemP) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) mma_ts2(tO, tP + kk * 8, v_lo + kk * (2048 >> 4), hi_k, idesc_pv, kk > 0 ? 1u : acc0);
            if (!mbar_wait(&bar_p[t], n_pv & 1, abort_v, 28)) break;
            tc_fence_after();
#pragma unroll
            for (int kk = 4; kk < kTile / 16; ++kk) mma_ts2(tO, tP + kk * 8, v_lo + kk * (2048 >> 4), hi_k, idesc_pv, 1u);
          } else {
#pragma unroll
            for (int kk = 0; kk < kTile / 16; ++kk) {
              const uint32_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
              mma_ss2(tO, p_lo + off, hi_k, v_lo + kk * (2048 >> 4), hi_k, idesc_pv, kk > 0 ? 1u : acc0);
            }
          }
          mma_commit(&bar_pv[t]);
          FTRACE(2 * t, n_pv, 3);
          ++n_pv;
          mma_commit(&bar_ring_free[slot]);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue: thread = query row of team t
    // One thread owns a whole score row: the row maximum and sum need no exchange between threads, and the 128
    // scores are read from tensor memory once and stay in registers, which frees the S columns for the next tile.
    fwd_reg_inc<216>();
    const int t = warp >> 2;
    const int row = tid & (kTile - 1);
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tSr = tmem + Cfg::score_col(t) + lane_base, tOr = tmem + Cfg::out_col(t) + lane_base, tPr = tmem + Cfg::p_col(t) + lane_base;
    uint8_t* sPt = sP + t * Cfg::kPBytes;
    uint32_t n_tiles = 0;  // tiles this team has processed so far
    uint32_t n_merged = 0; // query tiles that both teams had a part of
    FTRACE_ACC_DECL
    // The waits inside a tile are not asked how they ended: one that ran out has set the abort word, or found it set, for good, and
    // whatever is computed from there on stays in this CTA, because every warp looks at the word, as one, before an item's rows
    // leave.  A vote for each wait cost 5 % at D = 64 (causal 4k batch 4: 220 -> 232 us), a flag kept per lane 2 %.
    bool ok = true;
    constexpr int step = kShared ? 2 : 1;
    for (uint32_t it = 0; ok; ++it) {
      const uint32_t is = it % kFwdItemSlots;
      if (!mbar_wait_warp(&bar_item_full[is], (it / kFwdItemSlots) & 1, abort_v, 31)) break;
      const FwdItem& item = s_item[is];  // stays until the warp is through with it; what only the end of an item needs is read again there
      if (item.code < 0) break;
      auto done = [&]() {
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_item_empty[is]);
      };
      const int qb = kShared ? item.qb : item.qb + t, n = item.n[t];
      if (n == 0) {
        // No readable key tile: a defined result, nothing to compute.  (A second team without a part leaves that to the first.)
        const int q = qb * kTile + row;
        if (q < P.T && !(kShared && t == 1)) {
          __nv_bfloat16* orow = p.out + (size_t)item.b * p.o_sb + (size_t)item.h * p.o_sh + (size_t)q * p.o_st;
          for (int i = 0; i < D; i += 8) *reinterpret_cast<uint4*>(orow + i) = make_uint4(0, 0, 0, 0);
          p.lse[((size_t)item.b * p.H + item.h) * P.T + q] = -CUDART_INF_F;
        }
        done();
        continue;
      }
      const int32_t* list = P.fwd_idx + ((size_t)item.b * NB + qb) * NB + (kShared ? t : 0) + 2 * step;
      // List entries are fetched two tiles ahead and the mask of a partial tile one tile ahead, so that their latency
      // hides behind the sweeps of the tile before.
      int e_cur = item.first[t][0], e_nxt = item.first[t][1];
      // Row of the plan's mask table for this query row: the number of its run inside the tile.  Rows of runs past the
      // table, and all rows of sequences without one, work their masks out from the run lists (row_mask).
      // Rows past the sequence take the last run's masks: nothing of theirs is stored.
      uint32_t masks = kNoMasks;  // place in the table of this row's mask for key tile 0 (the table of as many batch elements as fit the card has fewer places)
      if (P.q_mask != nullptr) {
        int run = -1;
        const int nr = item.n_runs[t];
#pragma unroll
        for (int r = 0; r < kMaskRuns + 1; ++r)
          if (r < nr && item.runs[kShared ? 0 : t][r].start <= row) run = r;
        if (run < kMaskRuns) masks = (item.b * (uint32_t)(NB * (NB + 1) / 2) + (uint32_t)(qb * (qb + 1) / 2)) * kMaskRuns + run;
      }
      int4 mask_pf = make_int4(0, 0, 0, 0);
      auto prefetch_mask = [&](int entry) {
        if (entry & kFullBit) return;
        if (masks != kNoMasks) mask_pf = ld_nc_v4_here(P.q_mask + (masks + min((uint32_t)entry, (uint32_t)qb) * kMaskRuns));
      };
      prefetch_mask(e_cur);
      float m_used = -CUDART_INF_F, l = 0.f;
      FTRACE_ACC(0);
      if constexpr (!Cfg::kTmemP) {  // the store of the warp's last rows must have read their places, which are P's
        if (lane == 0) tma_store_wait_read0();
        __syncwarp();
      }
      for (int left = n; left > 0; --left) {
        const int entry = e_cur;
        e_cur = e_nxt;
        if (left > 2) e_nxt = ld_nc_i32_here(list);
        list += step;
        const int kb = entry & ~kFullBit;
        if ((uint32_t)kb >= (uint32_t)NB) { atomicCAS(abort_w, 0, 38); ok = false; break; }
        const int4 mask_cur = mask_pf;
        if (left > 1) prefetch_mask(e_cur);
        FTRACE_ACC(7);
        auto tile = [&](auto masked_tag) {
          constexpr bool kMasked = decltype(masked_tag)::value;
        uint32_t bits[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
        bool dead[4] = {false, false, false, false}, mixed[4] = {false, false, false, false};
        if (kMasked) {
          // 128-bit mask of the key columns this row may read, before causality
          if (masks != kNoMasks) {
            bits[0] = mask_cur.x; bits[1] = mask_cur.y; bits[2] = mask_cur.z; bits[3] = mask_cur.w;
          } else {
            const uint4 m4 = row_mask(P, p.mask, item.b, qb, kb, row);
            bits[0] = m4.x; bits[1] = m4.y; bits[2] = m4.z; bits[3] = m4.w;
          }
          if (kb == qb) {  // causal inside the diagonal tile: columns 0..row
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              const int hi = row + 1 - 32 * w;
              bits[w] &= hi >= 32 ? 0xffffffffu : (hi <= 0 ? 0u : ((1u << hi) - 1u));
            }
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {  // per 32-column chunk, uniform over the warp: nothing / everything / some allowed
            dead[c] = __all_sync(0xffffffffu, bits[c] == 0u);
            mixed[c] = !dead[c] && !__all_sync(0xffffffffu, bits[c] == 0xffffffffu);
          }
        }
        if (kMasked) FTRACE_ACC(1); else FTRACE_ACC(5);
        if (row == 0) FTRACE(2 * t + 1, n_tiles, 0);
        if (!mbar_try_wait(&bar_s[t], n_tiles & 1)) wait_longer(&bar_s[t], n_tiles & 1, abort_v, 32);
        tc_fence_after();
        FTRACE_ACC(2);
        if (row == 0) FTRACE(2 * t + 1, n_tiles, 1);
        uint32_t sv[4][32];
        tmem_ld32(tSr, sv[0]);
        tmem_ld32(tSr + 32, sv[1]);
        tmem_ld32(tSr + 64, sv[2]);
        tmem_ld32(tSr + 96, sv[3]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_sfree[t]);  // the issuer may now overwrite S with the next tile's scores
        if (row == 0) FTRACE(2 * t + 1, n_tiles, 2);
        // masked scores become -inf once; both sweeps below then need no mask (exp2(-inf) = 0)
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (kMasked && mixed[c]) {
#pragma unroll
            for (int i = 0; i < 32; ++i) sv[c][i] = ((bits[c] >> i) & 1u) ? sv[c][i] : 0xff800000u;
          }
        // sweep 1: row maximum (eight independent running maxima keep the dependency chain short)
        float mx8[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) mx8[i] = -CUDART_INF_F;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (!kMasked || !dead[c]) {
#pragma unroll
            for (int i = 0; i < 16; ++i) mx8[i & 7] = fmax3(mx8[i & 7], __uint_as_float(sv[c][i]), __uint_as_float(sv[c][i + 16]));
          }
        float mx = fmax3(fmax3(mx8[0], mx8[1], mx8[2]), fmax3(mx8[3], mx8[4], mx8[5]), fmaxf(mx8[6], mx8[7]));
        mx *= p.scale_log2;  // scale > 0, so max commutes with the scaling
        const float m_new = fmaxf(m_used, mx);
        const bool need = m_new > m_used + kRescaleThreshold || (m_used == -CUDART_INF_F && m_new > -CUDART_INF_F);
        const bool any_need = __any_sync(0xffffffffu, need);
        float factor = 1.f;
        if (any_need) {
          factor = need ? fast_exp2(m_used - m_new) : 1.f;  // exp2(-inf) = 0 on the first real tile
          l *= factor;
          if (need) m_used = m_new;
        }
        const float m_safe = m_used == -CUDART_INF_F ? 0.f : m_used;
        if (row == 0) FTRACE(2 * t + 1, n_tiles, 3);
        // sweep 2: P = exp2(s * scale - m) with packed fp32 arithmetic (two scores per instruction), row sum in
        // four partial sums, bf16 pack, P to its place
        const unsigned long long scale2 = pack_f32x2(p.scale_log2, p.scale_log2), negm2 = pack_f32x2(-m_safe, -m_safe);
        unsigned long long sum2[2] = {0ull, 0ull};
        uint32_t pk[4][16];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (!kMasked || !dead[c]) {
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              float x0, x1;
              unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[c][i]), __uint_as_float(sv[c][i + 1])), scale2, negm2), x0, x1);
              const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
              sum2[(i >> 1) & 1] = add_f32x2(sum2[(i >> 1) & 1], pack_f32x2(p0, p1));
              pk[c][i >> 1] = pack_bf16(p0, p1);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) pk[c][i] = 0u;
          }
          if (c == 1) {
            // P V of the previous tile must be complete before its P is overwritten and before O is touched;
            // it was issued a whole sweep ago, so this wait normally falls through.
            if (row == 0) FTRACE(2 * t + 1, n_tiles, 4);
            if (n_tiles > 0 && !mbar_try_wait(&bar_pv[t], (n_tiles - 1) & 1)) wait_longer(&bar_pv[t], (n_tiles - 1) & 1, abort_v, 33);
            tc_fence_after();  // P and O, both read or written by that product, are overwritten below
            if (row == 0) FTRACE(2 * t + 1, n_tiles, 5);
            if (any_need && left < n) {
              const unsigned long long f2 = pack_f32x2(factor, factor);
#pragma unroll 1
              for (int cc = 0; cc < D / 32; ++cc) {
                uint32_t r[32];
                tmem_ld32(tOr + cc * 32, r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                  float y0, y1;
                  unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), f2), y0, y1);
                  r[i] = __float_as_uint(y0);
                  r[i + 1] = __float_as_uint(y1);
                }
                tmem_st32(tOr + cc * 32, r);
              }
              tmem_st_wait();
            }
          }
          if constexpr (Cfg::kTmemP) {
            if (c == 1) tmem_st16(tPr, pk[0]);
            if (c >= 1) tmem_st16(tPr + 16 * c, pk[c]);
            if (c == 1) {
              tmem_st_wait();
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&bar_p0[t]);
            }
          } else if (c >= 1) {
#pragma unroll
            for (int cc = (c == 1 ? 0 : c); cc <= c; ++cc)
#pragma unroll
              for (int g = 0; g < 4; ++g)
                *reinterpret_cast<uint4*>(sPt + (cc >> 1) * 16384 + sw128_offset(row, (cc & 1) * 4 + g)) =
                    make_uint4(pk[cc][g * 4 + 0], pk[cc][g * 4 + 1], pk[cc][g * 4 + 2], pk[cc][g * 4 + 3]);
          }
        }
        {
          float s0, s1, s2, s3;
          unpack_f32x2(sum2[0], s0, s1);
          unpack_f32x2(sum2[1], s2, s3);
          l += (s0 + s1) + (s2 + s3);
        }
        if (row == 0) FTRACE(2 * t + 1, n_tiles, 6);
        if constexpr (Cfg::kTmemP) tmem_st_wait();
        else fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_p[t]);
        if (row == 0) FTRACE(2 * t + 1, n_tiles, 7);
        if (kMasked) FTRACE_ACC(6); else FTRACE_ACC(3);
        };
        if (entry & kFullBit) tile(std::false_type{}); else tile(std::true_type{});
        ++n_tiles;
      }
      if (!ok) break;
      // ---- epilogue: O / l -> bf16 -> the warp's rows of the team's buffer (at D = 128 P's, free after the last P V), 64 columns at a time ->
      //      TMA store.  A warp stores its own 32 rows, so that the team's warps need not meet.
      if (!(ok = __all_sync(0xffffffffu, mbar_wait(&bar_pv[t], (n_tiles - 1) & 1, abort_v, 34) && *abort_v == 0))) break;
      tc_fence_after();
      const int b = item.b, h = item.h, q = qb * kTile + row;
      const bool shared = kShared && item.n[1] > 0;  // both teams have a part of the query tile
      // Teams that share the query tile: team 1 leaves its part where it is, team 0 scales both to one maximum and adds them up.
      if (shared && t == 1) {
        s_merge[row] = make_float2(m_used, l);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_merge);
      } else {
        float f0 = 1.f, f1 = 0.f;
        if (shared) {
          if (!(ok = __all_sync(0xffffffffu, mbar_wait(bar_merge, n_merged & 1, abort_v, 35) && *abort_v == 0))) break;
          tc_fence_after();
          ++n_merged;
          const float2 other = s_merge[row];
          const float m = fmaxf(m_used, other.x);
          f0 = m_used == -CUDART_INF_F ? 0.f : fast_exp2(m_used - m);
          f1 = other.x == -CUDART_INF_F ? 0.f : fast_exp2(other.x - m);
          m_used = m;
          l = l * f0 + other.y * f1;
        }
        const float inv = l > 0.f ? 1.f / l : 0.f;
        f0 *= inv;
        f1 *= inv;
        if constexpr (Cfg::kTmemP) {  // the store of the warp's last rows must have read theirs
          if (lane == 0) tma_store_wait_read0();
          __syncwarp();
        }
#pragma unroll 1
        for (int s = 0; s < Cfg::kSub; ++s) {
          uint32_t o[2][32];
          tmem_ld32(tOr + s * 64, o[0]);
          tmem_ld32(tOr + s * 64 + 32, o[1]);
          if (shared) {
            uint32_t o1[2][32];
            tmem_ld32(tOr + Cfg::out_col(1) - Cfg::out_col(0) + s * 64, o1[0]);
            tmem_ld32(tOr + Cfg::out_col(1) - Cfg::out_col(0) + s * 64 + 32, o1[1]);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 64; ++i)
              o[i >> 5][i & 31] = __float_as_uint(__uint_as_float(o[i >> 5][i & 31]) * f0 + __uint_as_float(o1[i >> 5][i & 31]) * f1);
          } else {
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 64; ++i) o[i >> 5][i & 31] = __float_as_uint(__uint_as_float(o[i >> 5][i & 31]) * f0);
          }
          if (s == Cfg::kSub - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {  // the next item's first P V may overwrite O
              mbar_arrive(&bar_ofree[t]);
              if (shared) mbar_arrive(&bar_ofree[1]);
            }
          }
          uint8_t* box = sPt + s * 16384 + (warp & 3) * (32 * 128);
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const uint32_t* w = &o[g >> 2][(g & 3) * 8];
            uint4 v;
            v.x = pack_bf16(__uint_as_float(w[0]), __uint_as_float(w[1]));
            v.y = pack_bf16(__uint_as_float(w[2]), __uint_as_float(w[3]));
            v.z = pack_bf16(__uint_as_float(w[4]), __uint_as_float(w[5]));
            v.w = pack_bf16(__uint_as_float(w[6]), __uint_as_float(w[7]));
            *reinterpret_cast<uint4*>(box + sw128_offset(lane, g)) = v;
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) {
            const int first = qb * kTile + (warp & 3) * 32;
            if (first < P.T) tma_store_tile(&mapO, box, first, s, h, b);
            tma_store_commit();
          }
        }
        if (q < P.T) {
          // One rounding less where the sum is one of two parts, for those that adding them up takes: against 64 bits lse was 1-5 % further off
          // there than in a row that one team adds up (attention at T = 219 to 4096), and is 6-11 % closer now.
          constexpr float kLn2 = 0.6931471805599453f;
          p.lse[((size_t)b * p.H + h) * P.T + q] = l > 0.f ? (shared ? fmaf(m_used, kLn2, log2f(l) * kLn2) : (m_used + log2f(l)) * kLn2) : -CUDART_INF_F;
        }
      }
      done();
      FTRACE_ACC(4);
    }
    if (lane == 0) tma_store_wait_read0();  // the stores read this CTA's shared memory
    if (row == 0) FTRACE_CTA(2 + t, n_tiles);
    if (row == 0) FTRACE_ACC_DUMP(t);
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0) { FTRACE_SPAN(1); }
  if (*abort_v != 0) {
    // Let loads that were issued but never consumed land before the CTA's shared memory is released.
    if (tid == 0) atomicCAS(P.status, 0, 1000 + *abort_v);
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  if (warp == kFwdIssuerWarp) tmem_dealloc(tmem, 512);
  if (tid == 0) fwd_leave(P);
}

// Which work items a launch has: query tiles that the teams share, or pairs of query tiles or shared ones, whichever the lists call for.
enum FwdForm { kFwdPairs, kFwdShared, kFwdByLists };

// Every CTA comes to the same answer, because it depends on the plan and the grid (one CTA per SM) alone.  As pairs a launch that is short of items takes as long
// as its longest list, 2.0 us a tile.  As shared tiles it takes an SM's share of all lists, two tiles at a time in 1.65 us (D = 64; 1.8 us at D = 128, where two K/V
// streams do not fit the ring), and 3.2 us for each of the SM's items.  Shared tiles are taken where they come to less than 0.8 of the pairs' time: fitted to both forms
// of 330 random calls with more tiles than SMs and up to four pairs an SM; of 330 others it takes a form that is slower by more than 4 % six times, by 16 % at most.
// us, pairs | shared, each as a kernel of its own: linked 5133, H = 12, D = 128 63.6 | 52.3; 4 x 682, H = 12, D = 64 19.9 | 16.8; at the line documents 4 x 2639, H = 4, D = 64
// 20.8 | 20.0 and linked 8 x 608, H = 6, D = 128 17.3 | 17.9; beyond it linked 2 x 1278, H = 16, D = 64 24.3 | 26.3 and 4 x 8154, H = 3, D = 128 91.8 | 99.4.
// A kernel with both bodies runs the pairs 0.6 us slower than a kernel of its own, the shared tiles 1.2 us.
template <int D>
__device__ __forceinline__ bool lists_call_for_shared(const FwdParams& p, long long longest, long long all) {
  return (D == 64 ? 33 : 36) * all * p.H + 126ll * p.n_tiles < gridDim.x * (64 * longest + 30);
}

template <int D, int kForm>
__global__ void __launch_bounds__(kFwdThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapO, const __grid_constant__ FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  const FwdPlaces<D> at(smem_raw);
  const PlanView& P = p.plan;
  if (at.smem + FwdSmem<D>::kSmall + FwdSmem<D>::kSmallBytes > at.raw + FwdSmem<D>::kBytes) {  // a misplaced shared-memory window, the same in all CTAs: refused before anything is written there
    wait_previous();
    if (threadIdx.x == 0) atomicCAS(P.status, 0, 1901);
    return;
  }
  const uint32_t tmem = fwd_setup<D>(at);
  if (threadIdx.x == 0) FTRACE_SPAN(0);
  // What came before in the stream ends under the lines above; the plan is read from here on.
  wait_previous();
  int first[2] = {0, 0};
  if (threadIdx.x == kFwdProducerWarp * 32) {  // on their way while the plan's stamp is looked at; inside the plan's buffer whatever it holds
    int b, h;
    if (kForm != kFwdShared && static_cast<int>(blockIdx.x) < p.n_pairs) first[0] = ld_nc_i32_here(item_place(P, p.H, p.heads, p.head_group, false, blockIdx.x, b, h));
    if (kForm != kFwdPairs && static_cast<int>(blockIdx.x) < p.n_tiles) first[1] = ld_nc_i32_here(item_place(P, p.H, p.heads, p.head_group, true, blockIdx.x, b, h));
  }
  const int magic = P.status[kStampMagic], plan_b = P.status[kStampB], plan_t = P.status[kStampT], longest = P.status[kLongestList], all = P.status[kAllLists];
  const bool share = kForm == kFwdShared || (kForm == kFwdByLists && lists_call_for_shared<D>(p, longest, all));
  // Uniform across the grid: refuse a plan that was not built for this (B, T).  A CTA without an item leaves behind that, because a plan that is refused must not
  // keep a part of the count.
  const bool bad = magic != kPlanMagic || plan_b != P.B || plan_t != P.T;
  if (bad || static_cast<int>(blockIdx.x) >= (share ? p.n_tiles : p.n_pairs)) {
    if (threadIdx.x / 32 == kFwdIssuerWarp) tmem_dealloc(tmem, 512);
    if (threadIdx.x == 0) {
      if (bad) atomicCAS(P.status, 0, 1900);
      else fwd_leave(P);
    }
    return;
  }
  if (kForm == kFwdPairs || (kForm == kFwdByLists && !share)) fwd_items<D, false>(mapQ, mapK, mapV, mapO, p, at, tmem, first[0]);
  else fwd_items<D, true>(mapQ, mapK, mapV, mapO, p, at, tmem, first[1]);
}

// Host launcher.  Tensor strides are in elements; the last dimension is contiguous.
template <int D, int kForm>
static int launch_fwd_as(const void* q, const void* k, const void* v, void* out, float* lse, const int64_t* sq,
                         const int64_t* sk, const int64_t* sv, const int64_t* so, int B, int H, int T, float scale,
                        PlanView P, MaskArgs M, int sms, cudaStream_t stream) {
  CUtensorMap mq, mk, mv, mo;
  int r;
  if ((r = cached_tile_map(&mq, q, B, H, T, D, sq[0], sq[1], sq[2], kTile, D))) return r;
  if ((r = cached_tile_map(&mk, k, B, H, T, D, sk[0], sk[1], sk[2], kTile, D))) return r;
  if ((r = cached_tile_map(&mv, v, B, H, T, D, sv[0], sv[1], sv[2], kTile, D))) return r;
  if ((r = cached_tile_map(&mo, out, B, H, T, D, so[0], so[1], so[2], 32, 64))) return r;
  FwdParams p;
  p.plan = P; p.mask = M; p.lse = lse; p.out = static_cast<__nv_bfloat16*>(out);
  p.o_sb = so[0]; p.o_sh = so[1]; p.o_st = so[2];
  p.H = H; p.scale_log2 = scale * 1.4426950408889634f;
  p.n_pairs = B * H * ((P.NB + 1) / 2);
  p.n_tiles = B * H * P.NB;
  {  // heads per group, from the K and V bytes of one head (2 x T x D bf16 each)
    const long long kv_bytes = 4ll * T * D;
    long long g = (static_cast<long long>(TS2TS_FWD_GROUP_MB) << 20) / (kv_bytes > 0 ? kv_bytes : 1);
    p.heads = kv_bytes * B * H <= (static_cast<long long>(TS2TS_FWD_FOLD_MB) << 20) ? B * H : H;
    p.head_group = (int)(g < 1 ? 1 : (g > p.heads ? p.heads : g));
  }
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return -110;
  if (!attr_done[dev]) {
    if (cudaFuncSetAttribute(attn_fwd_kernel<D, kForm>, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdSmem<D>::kBytes) != cudaSuccess)
      return -110;
    attr_done[dev] = true;
  }
  const int most = kForm == kFwdPairs ? p.n_pairs : p.n_tiles;
  const unsigned grid = (unsigned)(most < sms ? most : sms);
  FTRACE_ATTACH(p, stream);
  cudaError_t launched;
  {
    ProfileScope timed(0, stream);
    launched = launch_after(attn_fwd_kernel<D, kForm>, dim3(grid), kFwdThreads, FwdSmem<D>::kBytes, stream, mq, mk, mv, mo, p);
  }
  FTRACE_DUMP(stream);
  const cudaError_t last = cudaGetLastError();
  return launched == cudaSuccess && last == cudaSuccess ? 0 : -111;
}

// Shared query tiles are twice as many and half as long, but bring in every key tile once a query tile instead of once a pair, which costs 10 % (D = 64) to 25 %
// (D = 128) where the launch is long enough to be bound by throughput (causal 4k batch 4, H = 16, D = 64 213 us as pairs, 234 shared; D = 128 282 and 350).  Where all of them run
// at once they always win (linked 600, H = 8, D = 64 13.1 -> 11.4; linked 1024, H = 4, D = 64 22.8 -> 16).  Up to four pairs an SM it depends on the lists, and the kernel
// looks at them; with more pairs the lists call for pairs (linked 4 x 17842, H = 2, D = 128, 3.8 an SM 242 as pairs, 250 shared; linked 2 x 14400, H = 8, D = 64, 6.2 an SM 269 and 275) or for neither
// (linked 16k, H = 12, D = 64, 5.2 an SM 252 and 249).
template <int D>
static int launch_fwd_t(const void* q, const void* k, const void* v, void* out, float* lse, const int64_t* sq, const int64_t* sk, const int64_t* sv,
                        const int64_t* so, int B, int H, int T, float scale, PlanView P, MaskArgs M, cudaStream_t stream) {
  static int sm_count[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return -110;
  if (sm_count[dev] <= 0 && (cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sm_count[dev] <= 0)) return -110;
  const int sms = sm_count[dev];
  const long long bh = (long long)B * H;
  const bool by_lists = bh * ((P.NB + 1) / 2) <= 4 * sms;
  const auto launch = bh * P.NB <= sms ? launch_fwd_as<D, kFwdShared> : by_lists ? launch_fwd_as<D, kFwdByLists> : launch_fwd_as<D, kFwdPairs>;
  return launch(q, k, v, out, lse, sq, sk, sv, so, B, H, T, scale, P, M, sms, stream);
}

int launch_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int64_t* sq, const int64_t* sk,
               const int64_t* sv, const int64_t* so, int B, int H, int T, int D, float scale, PlanView P, MaskArgs M,
               cudaStream_t stream) {
  if (D == 128) return launch_fwd_t<128>(q, k, v, out, lse, sq, sk, sv, so, B, H, T, scale, P, M, stream);
  if (D == 64) return launch_fwd_t<64>(q, k, v, out, lse, sq, sk, sv, so, B, H, T, scale, P, M, stream);
  return -112;
}

}  // namespace ts2ts
