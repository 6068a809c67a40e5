// sphg_movers.cuh -- the incremental re-sort: its record (written by the force
// pass, cleared by the density pass) and its launch interface (sphg_movers.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace sphg {

// Slots per block of the merge and per entry of the block sums.
constexpr int kMergeShift = 9;
constexpr int kMergeBlockSlots = 1 << kMergeShift;
// Blocks per entry of the second level of the sums (32,768 slots).
constexpr int kMergeSupShift = 6;
// Movers inserted before one slot, and into one block's slots: more than these
// make the iteration sort fully (a group is ordered pair by pair, a block's
// movers are held in shared memory).
constexpr int kGroupCap = 64;
constexpr int kBlockInsertCap = 512;
// The movers are counted in this many words, a cache line apart: atomics of a
// whole force pass on one word (or line) cost more than the pass itself.
constexpr int kMoverCounters = 8, kMoverCounterStride = 32;

// Where the force pass records the slots whose cell changed ("movers").  A
// mover's insertion point p in [0, n] is the number of current slots ordered
// before its (new key, slot); the movers of one p form a chain head[p] ->
// next[head[p]] -> ..., as long as the count says.  The counts and sums start at
// zero each iteration, so there are two copies of them: the force pass of step
// epoch e adds to copy (e + 1) & 1, which the next iteration's re-sort reads
// while it clears the other one.
struct MoverRecord {
  uint32_t* mask;     // [ceil(n/32)] bit s%32 of word s/32: slot s changed cell (every word written)
  uint32_t* head;     // [n+1] last mover recorded at p (valid where the count is not 0)
  uint32_t* next;     // [n] the one recorded before it
  uint32_t* counts;   // the two copies
  uint32_t* next_epoch;  // step epoch of the next iteration's cell ranges
  int64_t cap;        // particles a copy is laid out for
  const uint32_t* last;  // movers of the iteration before, and how many at most
  uint32_t record_limit; // for this one's to be recorded (record_limit())
};

// The parts of one copy, sized for cap particles.
struct MoverCounts {
  uint32_t* insc;     // movers inserted before slot p, one byte each, p in [0, n]
  int32_t* blk_net;   // [n/512 + 1] insertions - movers of each 512-slot block
  uint32_t* blk_ins;  // [n/512 + 1] insertions of each block
  int32_t* sup_net;   // [n/32768 + 1] insertions - movers of 64 blocks
  uint32_t* total;    // [kMoverCounters] movers, a line each; the first line's second word is
                      // set when a group or a block outgrew its cap (sort fully)
};
__host__ __device__ inline size_t mover_insc_words(int64_t cap) { return ((size_t)cap / 4 + 1 + 31) / 32 * 32; }
__host__ __device__ inline size_t mover_counts_words(int64_t cap) {
  const size_t nb = ((size_t)cap >> kMergeShift) + 1, ns = ((size_t)cap >> (kMergeShift + kMergeSupShift)) + 1;
  return mover_insc_words(cap) + (2 * nb + ns + 31) / 32 * 32 + kMoverCounters * kMoverCounterStride;
}
__host__ __device__ inline MoverCounts mover_counts(const MoverRecord& r, uint32_t copy) {
  const size_t nb = ((size_t)r.cap >> kMergeShift) + 1, ns = ((size_t)r.cap >> (kMergeShift + kMergeSupShift)) + 1;
  uint32_t* c = r.counts + (copy & 1u) * mover_counts_words(r.cap);
  MoverCounts m;
  m.insc = c;
  m.blk_net = reinterpret_cast<int32_t*>(c + mover_insc_words(r.cap));
  m.blk_ins = reinterpret_cast<uint32_t*>(m.blk_net + nb);
  m.sup_net = reinterpret_cast<int32_t*>(m.blk_ins + nb);
  m.total = c + mover_insc_words(r.cap) + (2 * nb + ns + 31) / 32 * 32;
  return m;
}

// Movers up to which an iteration merges, its record being there: small states a
// quarter (at least 8,192), larger ones any number -- us an iteration of random
// free particles, merge / full sort after the record: 423,000 particles 94 / 144
// with 28 % moving, 124 / 168 with 64 %; 2,000,000 382 / 494 and 533 / 631.  Either
// side of the line, with 23 % moving, merge / full sort without a record: 40,000
// 34.6 / 42.0, 60,000 38.3 / 47.8, 70,000 39.7 / 48.2, 131,072 45.9 / 60.5, 262,144
// 58.3 / 73.9; a full sort after the record takes 58 to 62 at 40,000 to 70,000.
inline int64_t mover_limit(int64_t n) {
  if (n > 65536) return n;
  return n / 4 > 8192 ? n / 4 : 8192;
}
// Movers of an iteration beyond which the next one's are counted but not
// recorded, and sorted fully: the record's atomics then cost more than the sort
// (2,000,000 particles: merge 298 us with 2 % moving, 335 with 14 %, 382 with 28 %,
// 447 with 44 %; full sort without a record 372).
inline int64_t record_limit(int64_t n) { return n > 65536 ? n / 3 : mover_limit(n); }

struct MoverArgs {
  int64_t n;
  int64_t limit;           // movers up to which the iteration merges
  MoverRecord rec;
  uint32_t* ctl;           // [0] = 1 when the merge ran, [1] = changed slots,
                           // [2] set to 1 if a record was inconsistent (never cleared here)
  uint32_t* epoch;         // step epoch of the cell-range table (set when the merge runs)
  const uint32_t* keyB;    // keys of the integrated state, previous slot order
  const float2* posB;
  const float2* velB;
  const int32_t* idsB;     // null when creation indices are not tracked
  uint32_t* keyA;          // out: sorted keys, state, creation indices
  float2* posA;
  float4* velpA;
  int32_t* idsA;
  uint32_t* perm;          // out: previous slot of each sorted position
  uint4* ranges;           // out: cell ranges {start, end, epoch, 0} of the sorted order
  unsigned long long cond; // graph conditional handle of the full sort (0: none), set to
                           // 1 when it must run, 0 when the merge handled the iteration
  int early_next;          // let the next kernel be scheduled at the start (allow_next_kernel)
};

// One launch: the decision (merge, or leave ctl[0] = 0 for the full sort), the
// sorted state and its cell ranges.
cudaError_t launch_movers(const MoverArgs& a, cudaStream_t st);

}  // namespace sphg
