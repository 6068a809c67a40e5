// sphg_lists.cu -- CSR neighbour lists of the current (sorted) state, in the
// reference's order: self included, stencil x offset outer, y offset inner,
// j ascending (MultipassNeighborLists: count CountNeighborsPerParticle
// core/algorithmic/MultipassNeighborLists.h:63-121, offsets CalculateOffsets
// :47-61, fill AssignIndices :123-181).  The reference GPU version
// (core/acceleration/cuNeighborLists.cu) drops the particle itself and leaves
// its index buffer uninitialised; this one follows the CPU semantics.
//
// One kernel: a block walks the stencil of its 128 particles once, each list
// kept in shared memory, scans the lengths, finds the entries before its own by
// a decoupled look-back over the preceding blocks' published totals, and writes
// offsets and entries -- packed for the passes of the lists mode, as plain
// indices, or ascending and delta-coded (Codifier::Encode).  Counting, a scan of
// three kernels and a second walk to fill took 30 us of an iteration of 93,623
// particles where this takes 17 (732 blocks, caches cold), and the export sorted and
// coded in two more.
#include <cstdint>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/sphg.h"
#include "sphg_neighbor.cuh"
#include "sphg_step.cuh"

namespace sphg {

constexpr int kListThreads = 128;
constexpr int kListWarps = kListThreads / 32;
constexpr int kListSlots = 32;  // entries of a list kept in shared memory; a longer list is walked again
constexpr int kListSpinLimit = 1 << 22;
// A block's word: the low bits of the launch's generation, a flag, a count.
constexpr int kCountBits = 42;
constexpr unsigned long long kCountMask = (1ull << kCountBits) - 1ull;
constexpr unsigned long long kOwn = 1ull << kCountBits;    // the block's own total
constexpr unsigned long long kUpTo = 2ull << kCountBits;   // the total up to its end
constexpr int kGenShift = kCountBits + 2;

// Delta-codes an ascending list in place: the first index verbatim, then
// idx[k] - idx[k-1] - 1 (Codifier::Encode, core/encoders/Encoder.h:27-44).
template <class Get, class Set>
__device__ __forceinline__ void delta_code(uint32_t n, Get&& get, Set&& set) {
  uint32_t prev = 0;
  for (uint32_t q = 0; q < n; ++q) {
    const uint32_t v = get(q);
    set(q, q ? v - prev - 1u : v);
    prev = v;
  }
}
// Insertion sort: lists hold a few dozen entries.
template <class Get, class Set>
__device__ __forceinline__ void sort_ascending(uint32_t n, Get&& get, Set&& set) {
  for (uint32_t q = 1; q < n; ++q) {
    const uint32_t v = get(q);
    uint32_t r = q;
    for (; r > 0 && get(r - 1) > v; --r) set(r, get(r - 1));
    set(r, v);
  }
}

template <int PREC, bool BATCHED, int FORM>
__global__ void __launch_bounds__(kListThreads) lists_assemble(StepArgs a, ListArgs o) {
  __shared__ uint32_t rec[kListSlots][kListThreads];
  __shared__ uint32_t s_blk, wsum[kListWarps];
  __shared__ unsigned long long s_before;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  cudaGridDependencySynchronize();
  if (skip_pass(a)) return;
  // blocks in the order they start: a look-back only waits on blocks that started earlier
  if (tid == 0) s_blk = atomicAdd(o.ctl, 1u);
  const unsigned long long gen = (unsigned long long)(*(volatile uint32_t*)(o.ctl + 1) & 0xfffffu) << kGenShift;
  __syncthreads();
  const uint32_t blk = s_blk;
  const int64_t i = (int64_t)blk * kListThreads + tid;
  auto entry = [](uint32_t j, uint32_t tag) { return FORM == kListPacked ? (j << 5) | tag : j; };
  auto walk = [&](auto&& put) {
    const InstDesc d = inst_of<BATCHED>(a, i);
    int cx, cy;
    uint32_t c = 0;
    for_each_neighbor<PREC, true>(a, d, a.keyA[i], a.posA[i], cx, cy,
                                  [&](uint32_t j, float, float, float, uint32_t tag) { put(c++, entry(j, tag)); });
    return c;
  };
  uint32_t c = 0;
  if (i < a.n)
    c = walk([&](uint32_t q, uint32_t e) {
      if (q < (uint32_t)kListSlots) rec[q][tid] = e;
    });
  // entries of the block's particles before this one, and of the block
  uint32_t x = c;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
    if (lane >= s) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  uint32_t excl = x - c, sum = 0;
#pragma unroll
  for (int w = 0; w < kListWarps; ++w) {
    excl += w < warp ? wsum[w] : 0u;
    sum += wsum[w];
  }
  if (warp == 0) {  // entries of the blocks before
    unsigned long long before = 0;
    if (lane == 0) atomicExch(o.words + blk, gen | (blk == 0 ? kUpTo : kOwn) | sum);
    int64_t t = (int64_t)blk - 1;
    int spins = 0;
    while (t >= 0) {
      const unsigned long long w = t - lane >= 0 ? *(volatile unsigned long long*)(o.words + (t - lane)) : gen | kUpTo;
      const bool ready = (w >> kGenShift) == (gen >> kGenShift) && (w & (kOwn | kUpTo));
      const unsigned missing = __ballot_sync(0xffffffffu, !ready);
      const unsigned whole = __ballot_sync(0xffffffffu, ready && (w & kUpTo));
      const int r = missing ? __ffs(missing) - 1 : 32, p = whole ? __ffs(whole) - 1 : 32;
      unsigned long long v = lane < r && lane <= p ? w & kCountMask : 0ull;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
      before += v;
      if (p < r) break;
      t -= r;
      if (r == 0) {
        if (++spins > kListSpinLimit) {  // give up: flag the error
          if (lane == 0) *(volatile uint32_t*)o.err = 1u;
          break;
        }
        __nanosleep(32);
      }
    }
    if (lane == 0) {
      if (blk) atomicExch(o.words + blk, gen | kUpTo | ((before + sum) & kCountMask));
      s_before = before;
    }
  }
  __syncthreads();
  if (i < a.n) {
    const int64_t base = (int64_t)(s_before + excl);
    o.offs[i] = base;
    if (i == a.n - 1) {
      o.offs[a.n] = base + c;
      if (o.total) *o.total = base + c;
    }
    if (o.idx) {
      uint32_t* out = o.idx + base;
      // entries past the buffer are not written, but reported
      const uint32_t room = base >= o.cap ? 0u : (uint32_t)min((int64_t)c, o.cap - base);
      if (room < c && o.overflow) *o.overflow = 1u;
      auto put = [&](uint32_t q, uint32_t e) {
        if (q < room) out[q] = e;
      };
      if (c <= (uint32_t)kListSlots) {
        auto get = [&](uint32_t q) { return rec[q][tid]; };
        if (FORM == kListCoded) {
          sort_ascending(c, get, [&](uint32_t q, uint32_t e) { rec[q][tid] = e; });
          delta_code(c, get, put);
        } else {
          for (uint32_t q = 0; q < c; ++q) put(q, get(q));
        }
      } else {
        walk(put);
        if (FORM == kListCoded && room == c) {
          auto get = [&](uint32_t q) { return out[q]; };
          sort_ascending(c, get, put);
          delta_code(c, get, put);
        }
      }
    }
  }
  if (tid == 0) {  // the last block leaves the counters for the next launch
    if (atomicAdd(o.ctl + 2, 1u) == gridDim.x - 1) {
      o.ctl[0] = 0u;
      o.ctl[2] = 0u;
      o.ctl[1] += 1u;
    }
  }
}

int64_t lists_blocks(int64_t n) { return (n + kListThreads - 1) / kListThreads; }

template <int FORM>
static cudaError_t assemble(const StepArgs& a, int precision, const ListArgs& o, cudaStream_t st) {
  const bool batched = (a.ninst > 1 || a.force_batched);
  const auto k = precision ? (batched ? lists_assemble<1, true, FORM> : lists_assemble<1, false, FORM>)
                           : (batched ? lists_assemble<0, true, FORM> : lists_assemble<0, false, FORM>);
  return launch_pdl(k, dim3((unsigned)lists_blocks(a.n)), dim3(kListThreads), 0, st, a, o);
}

cudaError_t launch_lists(const StepArgs& a, int precision, int form, const ListArgs& o, cudaStream_t st) {
  if (a.n == 0) return cudaSuccess;
  switch (form) {
    case kListPacked: return assemble<kListPacked>(a, precision, o, st);
    case kListCoded: return assemble<kListCoded>(a, precision, o, st);
    default: return assemble<kListIndices>(a, precision, o, st);
  }
}

// Delta codec of CSR lists (Codifier::Encode, core/encoders/Encoder.h:27-44):
// the first index of a list verbatim, then idx[k] - idx[k-1] - 1, which needs
// each list ascending.  One thread per list.
__global__ void delta_encode_kernel(const int64_t* offs, const int32_t* idx, int64_t n, int32_t* enc) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t b = offs[i], e = offs[i + 1];
  if (b >= e) return;
  int32_t prev = idx[b];
  enc[b] = prev;
  for (int64_t q = b + 1; q < e; ++q) {
    const int32_t v = idx[q];
    enc[q] = v - prev - 1;
    prev = v;
  }
}

__global__ void delta_decode_kernel(const int64_t* offs, const int32_t* enc, int64_t n, int32_t* out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t b = offs[i], e = offs[i + 1];
  if (b >= e) return;
  int32_t v = enc[b];
  out[b] = v;
  for (int64_t q = b + 1; q < e; ++q) {
    v = v + enc[q] + 1;
    out[q] = v;
  }
}

cudaError_t launch_delta(bool encode, const int64_t* offs, const int32_t* in, int64_t n, int32_t* out,
                         cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const unsigned g = (unsigned)((n + 255) / 256);
  if (encode) delta_encode_kernel<<<g, 256, 0, st>>>(offs, in, n, out);
  else delta_decode_kernel<<<g, 256, 0, st>>>(offs, in, n, out);
  return cudaGetLastError();
}


}  // namespace sphg
