// Layout of the block plan: the device buffer that the pre-pass fills from the
// per-token mask inputs and that the attention kernels read.  One plan serves
// every head and every layer of a micro-batch (the reference builds one
// BlockMask per micro-batch and broadcasts it, block_mask_creator.py:132-139).
//
// All tiles are 128 tokens.  NB = ceil(T / 128).
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <vector_types.h>

namespace ts2ts {

constexpr int kTile = 128;

enum : uint8_t { kSkip = 0, kPartial = 1, kFull = 2 };

// The backward gathers its query tiles from stretches of 32 query rows (see bwd_sub).  The plan's `state` byte of a tile pair
// holds in bits 0-3 which of the q tile's four stretches have an allowed (row, key) pair; kStateFull is set on top where every
// pair is allowed.  0 is a skipped pair.
constexpr int kStretch = 32, kStretches = kTile / kStretch;
constexpr uint8_t kStateFull = 0x80, kStateLive = 0x0f;
constexpr uint32_t kStretchFull = 0x8000u;  // in an entry of bwd_sub: the stretch belongs to a full tile

// A run is a maximal stretch of tokens inside one tile whose (doc id, row class,
// column class) triple is constant.  `start` is the offset inside the tile.
struct alignas(16) Run {
  int32_t start, doc, row, col;
};

constexpr uint32_t kFullBit = 1u << 30;  // set in merged list entries for full tiles

// Words of the status block.  Word 0 holds the first device error code.  The stamp is written by the pre-pass and
// compared by every attention kernel with its own B and T before it touches a list.  The ticket / done words are
// the work counters of the persistent attention kernels: a CTA draws work items from `ticket`; the last CTA to
// leave (counted in `done`) puts both back to zero, so launches that share a plan must be ordered on one stream.
enum : int {
  kStatusCode = 0, kStampMagic = 1, kStampB = 2, kStampT = 3,
  kLongestList = 4, kAllLists = 5,  // the forward's lists: the longest of the batch, and the sum of all of one head
  kFwdTicket = 8, kFwdDone = 9, kBwdTicket = 10, kBwdDone = 11,
  kLinkTRows = 12,  // > 0: link_t holds the transposed link bits of this many row classes
};
// Transposed link bits: word w of column class c holds, in bit r % 64, whether row class 64 w + r may read c.  A
// backward thread owns one key, i.e. one column class, and tests many row classes against it; with the transposed
// table its words are loaded once per CTA.  The table exists when R <= kLinkTMaxRows and 64 W <= kLinkTMaxCols.
constexpr int kLinkTMaxRows = 1024, kLinkTMaxCols = 1024, kLinkTWords = kLinkTMaxRows / 64;
// Masks of partial tiles, worked out once by the pre-pass for every head and layer: for tile pair (qb, kb) and each of the
// first kMaskRuns runs of the q tile the 128-bit mask of the key columns its rows may read (q_mask), and for each of the
// q tile's stretches and each of the first kMaskRuns runs of the kv tile the 32-bit mask of the query rows that may read its
// keys (kv_mask; 32 bytes a stretch, which one bulk copy takes along); causality inside the diagonal tile is left to the
// reader.  2 x 128 bytes a pair at or below the diagonal, so 8.4 MB a
// sequence of 32k; the tables exist up to kMaskMaxTiles tiles, and rows of later runs are worked out from the run lists.
constexpr int kMaskRuns = 8, kMaskMaxTiles = 512;
inline __host__ __device__ size_t mask_pair(int qb, int kb) { return (size_t)qb * (qb + 1) / 2 + kb; }

// Start of kv tile kb's line in a table with one slot for every q tile at or below the diagonal, lines one after the other.
inline __host__ __device__ size_t sub_line(int NB, int kb) { return (size_t)kb * NB - (size_t)kb * (kb - 1) / 2; }

constexpr int32_t kPlanMagic = 0x54533256;  // "TS2" and the layout's own mark: a plan of another layout is refused

struct PlanLayout {
  int B, T, NB;
  size_t status;      // int32[64]   see the kStatus* / kStamp* / k*Ticket words above
  size_t run_cnt;     // int32[B,NB]
  size_t runs;        // Run[B,NB,128]
  size_t state;       // uint8[B,NB,NB]   state[b,qb,kb], see kStateLive
  size_t fwd_cnt;     // int32[B,NB]      non-skipped kv tiles of q tile qb
  size_t fwd_idx;     // int32[B,NB,NB]   ascending kb, kFullBit set when full
  size_t bwd_cnt;     // int32[B,NB]      non-skipped q tiles of kv tile kb
  size_t bwd_idx;     // int32[B,NB,NB]   ascending qb, kFullBit set when full; written and read only where bwd_sub does not exist, idle space elsewhere
  size_t fwd_order;   // int32[B,NB]      q tiles of batch b by descending fwd_cnt
  size_t bwd_order;   // int32[B,NB]      kv tiles of batch b by descending bwd_tiles, or bwd_cnt where that does not exist
  size_t pair_cnt;    // int32[B,NP]      NP = ceil(NB/2): kv tiles that q tile 2p or 2p+1 reads (forward work items)
  size_t pair_order;  // int32[B,NP]      pairs of batch b by descending pair_cnt
  size_t link_t;      // uint64[B,kLinkTMaxCols,kLinkTWords]   transposed link bits (see kLinkTRows)
  size_t run_mask;    // uint32[B,NB,kMaskRuns,4]   the tokens of each of a tile's first runs, one bit a token
  size_t q_mask;      // uint32[B,NB(NB+1)/2,kMaskRuns,4]   see kMaskRuns; absent above kMaskMaxTiles
  size_t kv_mask;     // uint32[B,NB(NB+1)/2,kStretches,kMaskRuns]; absent above kMaskMaxTiles
  // The query tiles the backward walks for a kv tile, four stretches each.  Full q tiles come first, then partial ones whose
  // stretches are all live, each as it lies in memory; then the live stretches of the others, gathered, so that stretches without
  // an allowed pair take no part (linked 16k packs of the training sizes: 2743 tile pairs become 2450 tiles, of which 392 are gathered,
  // and 2657 become 2151; linked 32k, documents up to 2048, 15099 become 13458, up to 8192 13948 become 12828).  All ascend; the last tile is filled up with stretch number kStretches * NB, which lies past the sequence.
  size_t bwd_sub;     // uint16[B,NB(NB+1)/2,kStretches]   lines by sub_line(); stretch numbers
  size_t bwd_tiles;   // int32[B,NB]      tiles of each line; both absent above kMaskMaxTiles
  size_t bytes;
};

inline size_t plan_align(size_t x) { return (x + 255) & ~size_t(255); }

inline PlanLayout plan_layout(int B, int T) {
  PlanLayout L;
  L.B = B;
  L.T = T;
  L.NB = (T + kTile - 1) / kTile;
  const size_t nb = (size_t)L.NB, b = (size_t)B;
  size_t off = 0;
  L.status = off;    off = plan_align(off + 64 * sizeof(int32_t));
  L.run_cnt = off;   off = plan_align(off + b * nb * sizeof(int32_t));
  L.runs = off;      off = plan_align(off + b * nb * kTile * sizeof(Run));
  L.state = off;     off = plan_align(off + b * nb * nb);
  L.fwd_cnt = off;   off = plan_align(off + b * nb * sizeof(int32_t));
  L.fwd_idx = off;   off = plan_align(off + b * nb * nb * sizeof(int32_t));
  L.bwd_cnt = off;   off = plan_align(off + b * nb * sizeof(int32_t));
  L.bwd_idx = off;   off = plan_align(off + b * nb * nb * sizeof(int32_t));
  L.fwd_order = off; off = plan_align(off + b * nb * sizeof(int32_t));
  L.bwd_order = off; off = plan_align(off + b * nb * sizeof(int32_t));
  const size_t np = (nb + 1) / 2;
  L.pair_cnt = off;   off = plan_align(off + b * np * sizeof(int32_t));
  L.pair_order = off; off = plan_align(off + b * np * sizeof(int32_t));
  L.link_t = off;     off = plan_align(off + b * kLinkTMaxCols * kLinkTWords * sizeof(uint64_t));
  L.run_mask = off;   off = plan_align(off + b * nb * kMaskRuns * 16);
  const size_t masks = nb <= (size_t)kMaskMaxTiles ? b * (nb * (nb + 1) / 2) * kMaskRuns * 16 : 0;
  L.q_mask = off;     off = plan_align(off + masks);
  L.kv_mask = off;    off = plan_align(off + masks);
  L.bwd_sub = off;    off = plan_align(off + masks / (kMaskRuns * 16) * kStretches * sizeof(uint16_t));
  L.bwd_tiles = off;  off = plan_align(off + (masks > 0 ? b * nb * sizeof(int32_t) : 0));
  L.bytes = off;
  return L;
}

// Device-side view (pointers resolved from the layout).
struct PlanView {
  int B, T, NB;
  int32_t* status;
  int32_t* run_cnt;
  Run* runs;
  uint8_t* state;
  int32_t* fwd_cnt;
  int32_t* fwd_idx;
  int32_t* bwd_cnt;
  int32_t* bwd_idx;
  int32_t* fwd_order;
  int32_t* bwd_order;
  int32_t* pair_cnt;
  int32_t* pair_order;
  unsigned long long* link_t;
  uint4* run_mask;
  uint4* q_mask;   // nullptr when the tables do not exist, like the three after it
  uint32_t* kv_mask;
  uint16_t* bwd_sub;
  int32_t* bwd_tiles;
};

inline PlanView plan_view(void* base, int B, int T) {
  PlanLayout L = plan_layout(B, T);
  char* p = static_cast<char*>(base);
  PlanView v;
  v.B = B; v.T = T; v.NB = L.NB;
  v.status = reinterpret_cast<int32_t*>(p + L.status);
  v.run_cnt = reinterpret_cast<int32_t*>(p + L.run_cnt);
  v.runs = reinterpret_cast<Run*>(p + L.runs);
  v.state = reinterpret_cast<uint8_t*>(p + L.state);
  v.fwd_cnt = reinterpret_cast<int32_t*>(p + L.fwd_cnt);
  v.fwd_idx = reinterpret_cast<int32_t*>(p + L.fwd_idx);
  v.bwd_cnt = reinterpret_cast<int32_t*>(p + L.bwd_cnt);
  v.bwd_idx = reinterpret_cast<int32_t*>(p + L.bwd_idx);
  v.fwd_order = reinterpret_cast<int32_t*>(p + L.fwd_order);
  v.bwd_order = reinterpret_cast<int32_t*>(p + L.bwd_order);
  v.pair_cnt = reinterpret_cast<int32_t*>(p + L.pair_cnt);
  v.pair_order = reinterpret_cast<int32_t*>(p + L.pair_order);
  v.link_t = reinterpret_cast<unsigned long long*>(p + L.link_t);
  v.run_mask = reinterpret_cast<uint4*>(p + L.run_mask);
  v.q_mask = L.NB <= kMaskMaxTiles ? reinterpret_cast<uint4*>(p + L.q_mask) : nullptr;
  v.kv_mask = L.NB <= kMaskMaxTiles ? reinterpret_cast<uint32_t*>(p + L.kv_mask) : nullptr;
  v.bwd_sub = L.NB <= kMaskMaxTiles ? reinterpret_cast<uint16_t*>(p + L.bwd_sub) : nullptr;
  v.bwd_tiles = L.NB <= kMaskMaxTiles ? reinterpret_cast<int32_t*>(p + L.bwd_tiles) : nullptr;
  return v;
}

// Per-token mask inputs of one call (device pointers; row/col may alias doc).
struct MaskArgs {
  const int32_t* doc;    // [B,T]
  const int32_t* row;    // [B,T] row class of a query token, <0 = none
  const int32_t* col;    // [B,T] column class of a key token, <0 = none
  const int64_t* link;   // [B,R,W] bit c of row r: row class r may read column class c; nullptr = no links
  int R, W;
};

}  // namespace ts2ts
