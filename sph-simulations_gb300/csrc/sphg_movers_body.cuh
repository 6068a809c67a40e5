// sphg_movers_body.cuh -- the incremental re-sort's device code, shared by the
// stand-alone kernels (sphg_movers.cu: the merge; sphg_step.cu: the force
// pass's record) and the single-launch iteration (sphg_step.cu).  The algorithm
// is described in sphg_movers.cu.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

#include "sphg_common.cuh"
#include "sphg_movers.cuh"
#include "sphg_neighbor.cuh"
#include "sphg_step.cuh"

namespace sphg {

// Threads of a merge block: four slots each in the kernel of its own, whose many
// blocks hide each other's latency (eight warps of two slots: 1M dam break 81.8 ->
// 83.3 us an iteration, batch of 256 411 -> 420, 524,176 particles 48.5 -> 49.1,
// 262,144 32.6 -> 32.6, 512 x 512 vortex 37.1 -> 36.6, 131,044 25.3 -> 25.0, 93,636
// 25.0 -> 24.8, 40,000 21.0 -> 20.8); one each in the resident
// kernel, where a block has an SM's schedulers to itself and takes as long as its
// instructions (1,023 particles 11.7 -> 10.95 us, 6,084 28.1 -> 25.5, 12,800 16.6
// -> 16.2).
constexpr int kMergeThreads = 128;
constexpr int kResidentMergeThreads = 512;
constexpr int kMergeWords = kMergeBlockSlots / 32;  // mask words per block
static_assert(kMergeWords <= 32, "a warp scans the words");

// ---------------------------------------------------------------- the record
// Clears slot i's part of the copy the next force pass adds to (the reorder
// after a full sort; a merge clears its blocks' parts itself).
__device__ __forceinline__ void clear_mover_counts(const StepArgs& a, int64_t i, uint32_t epoch) {
  if (!a.movers.mask) return;
  const MoverCounts r = mover_counts(a.movers, epoch + 1u);
  const bool last = i == a.n - 1;  // also the entries of p = n
  if ((i & 3) == 0) r.insc[i >> 2] = 0u;
  if (last) r.insc[a.n >> 2] = 0u;
  for (int k = 0; k < 2; ++k) {
    const int64_t q = k == 0 ? i : a.n;
    if (k == 0 ? (i & (kMergeBlockSlots - 1)) != 0 : !last) continue;
    const int64_t b = q >> kMergeShift;
    r.blk_net[b] = 0;
    r.blk_ins[b] = 0u;
    r.sup_net[b >> kMergeSupShift] = 0;
  }
  if (i == 0)
    for (int k = 0; k < kMoverCounters; ++k) r.total[k * kMoverCounterStride] = r.total[k * kMoverCounterStride + 1] = 0u;
}

// The movers of one warp's 32 consecutive slots (bit l of moved: lane l's slot
// i moved to cell `key`) into the record.  The whole warp calls it.
__device__ __forceinline__ void record_movers(const StepArgs& a, uint32_t i, uint32_t key, unsigned moved) {
  const uint32_t epoch = *a.epoch;
  const MoverCounts r = mover_counts(a.movers, epoch + 1u);
  const int lane = threadIdx.x & 31;
  const bool mine = (moved >> lane) & 1u;
  if (lane == __ffs(moved) - 1)
    atomicAdd(r.total + ((i >> 5) % kMoverCounters) * kMoverCounterStride, (uint32_t)__popc(moved));
  if (*a.movers.last > a.movers.record_limit) {  // many moved the last time: sort fully
    if (lane == 0) r.total[1] = 1u;
    return;
  }
  // insertion point: the new cell's range when it holds particles now (the slot
  // itself is not among them), else a warp-wide 32-way search of the keys, once for
  // every cell of the warp's movers (32 of 30,000 particles into one empty cell:
  // 29.3 us an iteration, searched for one by one 43.3)
  uint32_t p = 0;
  bool search = false;
  if (mine) {
    const uint4 cr = a.ranges[key];
    search = cr.z != epoch || cr.x >= cr.y;
    p = i < cr.x ? cr.x : cr.y;
  }
  for (unsigned todo = __ballot_sync(0xffffffffu, search); todo;) {
    const uint32_t k = __shfl_sync(0xffffffffu, key, __ffs(todo) - 1);
    int64_t lo = 0, hi = a.n;
    while (hi > lo) {
      const int64_t step = (hi - lo + 31) / 32;
      const int64_t q = lo + (int64_t)(lane + 1) * step - 1;
      const int c = __popc(__ballot_sync(0xffffffffu, q < hi && a.keyA[q] < k));
      const int64_t nhi = lo + (int64_t)(c + 1) * step - 1;
      lo += (int64_t)c * step;
      if (nhi < hi) hi = nhi;
      if (lo > hi) lo = hi;
    }
    const bool found = search && key == k;
    if (found) p = (uint32_t)lo;
    todo &= ~__ballot_sync(0xffffffffu, found);
  }
  if (mine && p <= (uint64_t)a.n) {
    const int sh = 8 * (int)(p & 3u);
    const uint32_t before = (atomicAdd(r.insc + (p >> 2), 1u << sh) >> sh) & 255u;
    const uint32_t in_block = atomicAdd(r.blk_ins + (p >> kMergeShift), 1u);
    a.movers.next[i] = atomicExch(a.movers.head + p, i);
    // net changes: most movers stay in their block of slots, nearly all in the 64 blocks
    const uint32_t bp = p >> kMergeShift, bi = i >> kMergeShift;
    if (bp != bi) {
      atomicAdd(r.blk_net + bp, 1);
      atomicSub(r.blk_net + bi, 1);
      if (bp >> kMergeSupShift != bi >> kMergeSupShift) {
        atomicAdd(r.sup_net + (bp >> kMergeSupShift), 1);
        atomicSub(r.sup_net + (bi >> kMergeSupShift), 1);
      }
    }
    if (before >= (uint32_t)kGroupCap || in_block >= (uint32_t)kBlockInsertCap) r.total[1] = 1u;
  }
}

// ---------------------------------------------------------------- the merge
// The decision, from the force pass's record: merge when at most `limit` slots
// changed and no cap was passed.
// (The whole warp calls it.)
__device__ __forceinline__ bool merge_wanted(const MoverArgs& a, const uint32_t* total, uint32_t* movers) {
  const int lane = threadIdx.x & 31;
  const volatile uint32_t* t = total;
  const uint32_t m = lane < kMoverCounters ? t[lane * kMoverCounterStride] : 0u, capped = t[1];
  *movers = __reduce_add_sync(0xffffffffu, m);
  return (int64_t)*movers <= a.limit && capped == 0u;
}
// The leader's part of it: the decision word, the count, the step
// epoch, the graph's conditional.
__device__ __forceinline__ void merge_decided(const MoverArgs& a, bool merge, uint32_t movers, uint32_t epoch) {
  a.ctl[0] = merge ? 1u : 0u;
  a.ctl[1] = movers;
  if (merge) *a.epoch = epoch;
  if (a.cond) cudaGraphSetConditional((cudaGraphConditionalHandle)a.cond, merge ? 0u : 1u);
}

__device__ __forceinline__ uint32_t merge_inserted(const uint32_t* insc, int64_t p) {
  return reinterpret_cast<const uint8_t*>(insc)[p];
}

// Smallest or largest key among the c movers inserted before slot p.
__device__ __forceinline__ uint32_t merge_group_key(const MoverArgs& a, int64_t p, uint32_t c, bool largest) {
  uint32_t m = a.rec.head[p], k = largest ? 0u : kNoIndex;
  for (uint32_t q = 0; q < c && m < a.n; ++q) {
    const uint32_t km = a.keyB[m];
    k = largest ? max(k, km) : min(k, km);
    m = a.rec.next[m];
  }
  return k;
}

// Key of the last element of the sorted order that comes before the insertions
// of slot `base` (a multiple of 32), kNoIndex if none.  The whole warp calls it.
__device__ __forceinline__ uint32_t merge_prev_key(const MoverArgs& a, const uint32_t* insc, int64_t base, int lane) {
  for (int64_t q = base - 32; q >= 0; q -= 32) {
    const int64_t i = q + lane;
    const bool stay = !((a.rec.mask[q >> 5] >> lane) & 1u);
    const uint32_t c = merge_inserted(insc, i);
    const unsigned b = __ballot_sync(0xffffffffu, stay || c);
    if (!b) continue;
    const int l = 31 - __clz(b);
    uint32_t k = 0;
    if (lane == l) k = stay ? a.keyB[i] : merge_group_key(a, i, c, true);
    return __shfl_sync(0xffffffffu, k, l);
  }
  return kNoIndex;
}

// Key of the first element from slot q on (its insertions included), kNoIndex if none.
__device__ __forceinline__ uint32_t merge_next_key(const MoverArgs& a, const uint32_t* insc, int64_t from, int lane) {
  for (int64_t q = from; q <= a.n; q += 32) {
    const int64_t i = q + lane;
    const bool stay = i < a.n && !((a.rec.mask[q >> 5] >> lane) & 1u);
    const uint32_t c = i <= a.n ? merge_inserted(insc, i) : 0u;
    const unsigned b = __ballot_sync(0xffffffffu, stay || c);
    if (!b) continue;
    const int l = __ffs(b) - 1;
    uint32_t k = 0;
    if (lane == l) k = c ? merge_group_key(a, i, c, false) : a.keyB[i];
    return __shfl_sync(0xffffffffu, k, l);
  }
  return kNoIndex;
}

// Stores of data that a later phase of the same launch reads (kFused) bypass L1.
template <int LAUNCH, class V>
__device__ __forceinline__ void merge_store(V* p, V v) {
  if constexpr (LAUNCH == kFused) __stcg(p, v);
  else *p = v;
}

// The barrier of a merge block's threads: a thread block, or one of several in
// the resident kernel's blocks.
template <int LAUNCH, int THREADS>
__device__ __forceinline__ void merge_sync() {
  if constexpr (LAUNCH == kResident)
    asm volatile("barrier.sync %0, %1;" ::"r"(1u + threadIdx.x / THREADS), "n"(THREADS) : "memory");
  else __syncthreads();
}

struct MergeShared {
  uint32_t stay[kMergeWords];            // bit per slot: it keeps its cell
  uint32_t tot[kMergeWords];             // stayers + insertions of the word | insertions << 16
  int32_t red[kResidentMergeThreads / 32];
  bool merge;
  uint32_t prev, next;                   // keys either side of the block's output
  uint32_t ikey[kBlockInsertCap], islot[kBlockInsertCap];
  uint32_t igrp[kBlockInsertCap];        // first list entry of the mover's group << 16 | its size
  uint32_t iout[kBlockInsertCap];        // block-local output position of its group
  uint32_t key[kMergeBlockSlots + kBlockInsertCap];  // the block's output keys
};

// Merge block blk: the movers inserted before slots [512 blk, 512 blk + 512)
// and the slots themselves that keep their cell, to one contiguous run of the
// sorted order, with the cell ranges; and the block's part of the other copy of
// the counts cleared.  Returns false, having written nothing, when the record
// says to sort fully (the block of slot 0 records the decision either way).
// Every thread of the block calls it; epoch: *rec.next_epoch.  What bounds it is latency -- a block
// goes from its loads through two or four barriers to its stores -- so every
// load that needs no other is issued at the top, before the decision is known.
template <int LAUNCH, int THREADS = kMergeThreads>
__device__ __forceinline__ bool merge_block(const MoverArgs& a, MergeShared& sh, int64_t blk, uint32_t epoch) {
  constexpr int kSlots = kMergeBlockSlots / THREADS, kWarps = THREADS / 32;  // slots per thread
  static_assert(kWarps >= 4, "warp 1 decides, warps 2 and 3 find the neighbours");
  const int tid = threadIdx.x & (THREADS - 1), lane = tid & 31, warp = tid >> 5;
  const int64_t base = blk << kMergeShift;
  const unsigned lt = (1u << lane) - 1u;
  uint32_t key[kSlots], mw[kSlots];
  float2 p[kSlots], v[kSlots];
  int32_t id[kSlots];
#pragma unroll
  for (int u = 0; u < kSlots; ++u) {
    const int64_t i = base + (u * kWarps + warp) * 32 + lane;
    const bool in = i < a.n;
    mw[u] = in ? a.rec.mask[i >> 5] : ~0u;
    key[u] = in ? a.keyB[i] : 0u;
    p[u] = in ? a.posB[i] : make_float2(0.f, 0.f);
    v[u] = in ? a.velB[i] : make_float2(0.f, 0.f);
    id[u] = in && a.idsA ? a.idsB[i] : 0;
  }
  // the slots either side of the block, which nearly always decide its neighbours' keys
  const int64_t side = warp == 2 ? base - 1 : base + kMergeBlockSlots;
  const bool has_side = (warp == 2 || warp == 3) && side >= 0 && side < a.n;
  const uint32_t side_mask = has_side ? a.rec.mask[side >> 5] : 0u;
  const uint32_t side_key = has_side ? a.keyB[side] : 0u;
  const MoverCounts r = mover_counts(a.rec, epoch);
  if (warp == 1) {
    uint32_t movers;
    const bool merge = merge_wanted(a, r.total, &movers);
    if (lane == 0) {
      sh.merge = merge;
      if (blk == 0) merge_decided(a, merge, movers, epoch);
    }
  }
  uint32_t c[kSlots], cex[kSlots];
#pragma unroll
  for (int u = 0; u < kSlots; ++u) {
    const int64_t i = base + (u * kWarps + warp) * 32 + lane;
    c[u] = i <= a.n ? merge_inserted(r.insc, i) : 0u;
  }
  const uint32_t side_ins = has_side ? merge_inserted(r.insc, side) : 0u;
  // slots before the block whose movers left, movers inserted before it
  int32_t d = 0;
  const int64_t sup = blk >> kMergeSupShift, b0 = sup << kMergeSupShift;
  for (int64_t q = tid; q < sup; q += THREADS) d += r.sup_net[q];
  if (tid < blk - b0) d += r.blk_net[b0 + tid];
  if (warp == 2) {
    uint32_t k = kNoIndex;
    if (has_side) {
      k = side_key;
      if ((side_mask >> (side & 31)) & 1u) k = merge_prev_key(a, r.insc, base, lane);
    }
    if (lane == 0) sh.prev = k;
  } else if (warp == 3) {
    uint32_t k = side_key;
    if (!has_side || side_ins || ((side_mask >> (side & 31)) & 1u)) k = merge_next_key(a, r.insc, side, lane);
    if (lane == 0) sh.next = k;
  }
  bool stay[kSlots];
#pragma unroll
  for (int u = 0; u < kSlots; ++u) {
    const int w = u * kWarps + warp;
    stay[u] = !((mw[u] >> lane) & 1u);
    const unsigned sb = __ballot_sync(0xffffffffu, stay[u]);
    uint32_t incl = c[u];
    if (__any_sync(0xffffffffu, c[u] != 0u)) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
    }
    cex[u] = incl - c[u];
    if (lane == 31) {
      sh.stay[w] = sb;
      sh.tot[w] = ((uint32_t)__popc(sb) + incl) | (incl << 16);
    }
  }
  d = __reduce_add_sync(0xffffffffu, d);
  if (lane == 0) sh.red[warp] = d;
  merge_sync<LAUNCH, THREADS>();
  if (!sh.merge) return false;
  {  // the other copy, which this iteration's force pass adds to
    const MoverCounts o = mover_counts(a.rec, epoch + 1u);
    if (tid < kMergeBlockSlots / 4 && base + 4 * tid <= a.n) o.insc[(base >> 2) + tid] = 0u;
    if (tid == 0) {
      o.blk_net[blk] = 0;
      o.blk_ins[blk] = 0u;
      if (blk == b0) o.sup_net[sup] = 0;
    }
    if (blk == 0 && tid < kMoverCounters)
      o.total[tid * kMoverCounterStride] = o.total[tid * kMoverCounterStride + 1] = 0u;
  }
  // the same of the words before each word (every warp scans the block's words)
  uint32_t off, all;
  {
    const uint32_t t = lane < kMergeWords ? sh.tot[lane] : 0u;
    uint32_t incl = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    off = incl - t;
    all = __shfl_sync(0xffffffffu, incl, 31);
  }
  int64_t out0 = base;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) out0 += sh.red[w];
  const uint32_t total = all & 0xffffu, nins = all >> 16;
  // a consistent record stays inside the buffers; anything else is reported, not written
  if (out0 < 0 || out0 + (int64_t)total > a.n || nins > (uint32_t)kBlockInsertCap) {
    if (tid == 0) a.ctl[2] = 1u;
    merge_sync<LAUNCH, THREADS>();
    return true;
  }
#pragma unroll
  for (int u = 0; u < kSlots; ++u) {
    const int w = u * kWarps + warp;
    const int64_t i = base + w * 32 + lane;
    const uint32_t woff = __shfl_sync(0xffffffffu, off, w);
    const uint32_t grp = (woff & 0xffffu) + (uint32_t)__popc(sh.stay[w] & lt) + cex[u];
    if (stay[u]) {
      const uint32_t q = grp + c[u];
      const int64_t to = out0 + q;
      sh.key[q] = key[u];
      merge_store<LAUNCH>(a.posA + to, p[u]);
      merge_store<LAUNCH>(a.velpA + to, make_float4(v[u].x, v[u].y, 0.f, 0.f));
      merge_store<LAUNCH>(a.perm + to, (uint32_t)i);
      if (a.idsA) merge_store<LAUNCH>(a.idsA + to, id[u]);
    }
    if (c[u]) {  // the movers inserted before slot i, in any order
      const uint32_t l0 = (woff >> 16) + cex[u];
      uint32_t m = a.rec.head[i];
      for (uint32_t q = 0; q < c[u]; ++q) {
        const bool ok = m < a.n;
        sh.islot[l0 + q] = ok ? m : kNoIndex;
        sh.ikey[l0 + q] = ok ? a.keyB[m] : 0u;
        sh.igrp[l0 + q] = (l0 << 16) | c[u];
        sh.iout[l0 + q] = grp;
        if (ok) m = a.rec.next[m];
      }
    }
  }
  merge_sync<LAUNCH, THREADS>();
  if (nins) {
  for (uint32_t q = tid; q < nins; q += THREADS) {
    const uint32_t k = sh.ikey[q], s = sh.islot[q], g = sh.igrp[q];
    uint32_t rank = 0;  // among its group, by (key, slot)
    for (uint32_t r = g >> 16, e = r + (g & 0xffffu); r < e; ++r)
      rank += sh.ikey[r] < k || (sh.ikey[r] == k && sh.islot[r] < s);
    const uint32_t at = sh.iout[q] + rank;
    if (s >= a.n || at >= total) {
      a.ctl[2] = 1u;
      continue;
    }
    const int64_t to = out0 + at;
    sh.key[at] = k;
    const float2 vm = a.velB[s];
    merge_store<LAUNCH>(a.posA + to, a.posB[s]);
    merge_store<LAUNCH>(a.velpA + to, make_float4(vm.x, vm.y, 0.f, 0.f));
    merge_store<LAUNCH>(a.perm + to, s);
    if (a.idsA) merge_store<LAUNCH>(a.idsA + to, a.idsB[s]);
  }
  merge_sync<LAUNCH, THREADS>();
  }
  uint32_t* rg = reinterpret_cast<uint32_t*>(a.ranges);
  for (uint32_t q = tid; q < total; q += THREADS) {
    const uint32_t k = sh.key[q];
    const uint32_t kp = q ? sh.key[q - 1] : sh.prev, kn = q + 1 < total ? sh.key[q + 1] : sh.next;
    const uint32_t i = (uint32_t)(out0 + q);
    merge_store<LAUNCH>(a.keyA + i, k);
    if (k != kp) {
      merge_store<LAUNCH>(rg + 4 * (size_t)k, i);
      merge_store<LAUNCH>(rg + 4 * (size_t)k + 2, epoch);
    }
    if (k != kn) merge_store<LAUNCH>(rg + 4 * (size_t)k + 1, i + 1u);
  }
  merge_sync<LAUNCH, THREADS>();  // (a block calling again reuses the shared arrays)
  return true;
}

}  // namespace sphg
