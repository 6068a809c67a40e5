// sphg_sort.cu -- stable LSD radix sort of (uint32 key, uint32 value) pairs,
// written for this library (no CUB/Thrust).  It replaces the
// thrust::sort_by_key of cuSortContainerByCellID
// (core/acceleration/cuFindNeighbors.cu:82-100), sorting the slot index
// instead of six payload arrays; the payload is gathered once afterwards.
//
// One-sweep structure, 8-bit digits:
//   sort_hist_all   one read of the keys -> digit histograms of every pass
//   sort_pass       one kernel per pass: a CTA takes the next tile of 2,048 or
//                   4,096 keys (tile ids handed out in start order by an atomic
//                   counter); each warp ranks its own run of consecutive keys
//                   stably against counters of its own (__match_any_sync +
//                   popc, no block barrier), the CTA adds the warps up, publishes
//                   its per-digit counts, puts the pairs in digit order in
//                   shared memory, finds its global offsets by a decoupled
//                   look-back over the preceding tiles' published counts
//                   (sixteen a round trip), and writes runs of equal digits.
// The look-back only waits on tiles that started earlier (so it cannot
// deadlock); each wait is bounded and sets an error word if it gives up.
//
// What bounds a pass is the chain tile id -> keys -> ranks -> look-back -> writes
// of each CTA, not its 16 bytes a pair.
#include <cstdint>
#include <cuda_runtime.h>

#include "sphg_common.cuh"
#include "sphg_sort.cuh"

namespace sphg {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kTile = kSortThreads * kSortItems;
constexpr int kRadix = 256;
constexpr int kWarps = kSortThreads / 32;
constexpr int kMaxPasses = 4;
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagPre = 2u << 30;
constexpr uint32_t kValMask = kFlagAgg - 1u;
constexpr int kSpinLimit = 1 << 22;

static inline int passes_for(int bits) { return bits <= 0 ? 1 : (bits + 7) / 8; }

int sort_num_tiles(int64_t n) { return (int)((n + kTile - 1) / kTile); }

// scratch: [error word][pad to 256 - passes][passes x 256 histogram][passes tile
//          counters][passes x ntiles x 256 look-back words]
static inline size_t head_words() { return (size_t)kMaxPasses * kRadix + 256; }

size_t sort_scratch_words(int64_t n) {
  return head_words() + (size_t)kMaxPasses * kRadix * (size_t)sort_num_tiles(n);
}
static_assert(kMaxPasses * kRadix + 256 == 1280 && kTile == 2048, "sort_scratch_words_c layout");

// Digit histograms of every pass in one read of the keys.  Each thread counts
// a run of 16 consecutive keys; nearly sorted input has long runs of equal
// digits, so one shared atomic per run and pass replaces one per key.
constexpr int kHistPerThread = 16;

__global__ void __launch_bounds__(kSortThreads) sort_hist_all(const uint32_t* __restrict__ keys,
                                                              int64_t n, int passes,
                                                              uint32_t* __restrict__ ghist,
                                                              const uint32_t* skip) {
  __shared__ uint32_t h[kMaxPasses][kRadix];
  for (int p = 0; p < kMaxPasses; ++p) h[p][threadIdx.x] = 0;
  cudaGridDependencySynchronize();
  if (skip && *skip) return;
  __syncthreads();
  const int64_t chunk = (int64_t)kSortThreads * kHistPerThread;
  for (int64_t b = (int64_t)blockIdx.x * chunk; b < n; b += (int64_t)gridDim.x * chunk) {
    const int64_t s0 = b + (int64_t)threadIdx.x * kHistPerThread;
    uint32_t k[kHistPerThread];
    // 16-byte loads only where the address allows them: a caller's buffer may
    // start at any 4-byte boundary (a view such as keys + 1)
    if (s0 + kHistPerThread <= n && ((reinterpret_cast<uintptr_t>(keys + s0) & 15u) == 0)) {
#pragma unroll
      for (int q = 0; q < kHistPerThread; q += 4) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(keys + s0 + q));
        k[q] = v.x; k[q + 1] = v.y; k[q + 2] = v.z; k[q + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < kHistPerThread; ++q) k[q] = s0 + q < n ? __ldg(keys + s0 + q) : 0u;
    }
    const int m = (int)(s0 >= n ? 0 : (n - s0 < kHistPerThread ? n - s0 : kHistPerThread));
    for (int p = 0; p < passes; ++p) {
      uint32_t run_d = 0, run_c = 0;
#pragma unroll
      for (int q = 0; q < kHistPerThread; ++q) {
        if (q >= m) break;
        const uint32_t d = (k[q] >> (8 * p)) & (kRadix - 1);
        if (run_c && d != run_d) {
          atomicAdd(&h[p][run_d], run_c);
          run_c = 0;
        }
        run_d = d;
        ++run_c;
      }
      if (run_c) atomicAdd(&h[p][run_d], run_c);
    }
  }
  __syncthreads();
  for (int p = 0; p < passes; ++p)
    if (h[p][threadIdx.x]) atomicAdd(&ghist[p * kRadix + threadIdx.x], h[p][threadIdx.x]);
}

// Exclusive scan of one value per thread over the CTA.
__device__ __forceinline__ uint32_t cta_excl_scan(uint32_t v, uint32_t* wsum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  uint32_t e = x - v;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) e += w < warp ? wsum[w] : 0u;
  return e;
}

// Lanes of the warp whose digit equals the caller's (d in [0, 256], 256: none),
// by a ballot per bit: __match_any_sync takes a step per distinct value, and
// 32 random digits are nearly all distinct.
__device__ __forceinline__ unsigned digit_peers(uint32_t d) {
  unsigned peers = __ballot_sync(0xffffffffu, d < (uint32_t)kRadix);
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const unsigned m = __ballot_sync(0xffffffffu, (d >> b) & 1u);
    peers &= ((d >> b) & 1u) ? m : ~m;
  }
  return peers;
}

template <int ITEMS, bool VALS>
__global__ void __launch_bounds__(kSortThreads, 4) sort_pass(  // four a SM: 64 registers (20M pairs 842 -> 593 us)
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
    uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int64_t n, int pass,
    const uint32_t* __restrict__ ghist, uint32_t* tile_counter, uint32_t* lookback,
    uint32_t* err, uint32_t* epoch, const uint32_t* skip) {
  static_assert(kSortThreads == kRadix, "one thread per digit");
  constexpr int kTileKeys = kSortThreads * ITEMS;
  __shared__ uint32_t s_tile, s_wsum[2][kWarps];
  __shared__ uint32_t s_base[kRadix];          // output position of a digit's first key less its place in the tile
  __shared__ uint32_t s_cnt[kWarps][kRadix];   // per warp: keys of each digit, then its first one's place in the tile
  __shared__ uint32_t s_key[kTileKeys], s_val[kTileKeys];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int shift = 8 * pass;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) s_cnt[w][tid] = 0;
  cudaGridDependencySynchronize();  // the pass before
  if (skip && *skip) return;        // the incremental re-sort handled this step
  if (tid == 0) s_tile = atomicAdd(tile_counter + pass, 1u);
  const uint32_t tot = ghist[pass * kRadix + tid];
  __syncthreads();
  const uint32_t tile = s_tile;
  const int64_t base = (int64_t)tile * kTileKeys;
  if (epoch && tile == 0 && tid == 0) *epoch += 1u;  // nobody reads the epoch during the sort

  // the warp's run of consecutive keys, 32 a round
  uint32_t key[ITEMS];
  uint32_t rank2[ITEMS / 2];  // places below 4,096, two a register
  const int64_t i0 = base + (int64_t)warp * (32 * ITEMS) + lane;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const int64_t i = i0 + k * 32;
    key[k] = i < n ? __ldg(keys_in + i) : 0u;
  }
  // start of digit tid in the output: exclusive scan of this pass's histogram
  const uint32_t dstart = cta_excl_scan(tot, s_wsum[0]);
  // stable ranks within the warp's run
  const unsigned lt_mask = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const bool valid = i0 + k * 32 < n;
    const uint32_t d = valid ? (key[k] >> shift) & (kRadix - 1) : kRadix;
    const unsigned peers = digit_peers(d);
    uint32_t before = 0;
    if (valid) before = s_cnt[warp][d];
    const uint32_t r = before + __popc(peers & lt_mask);
    rank2[k / 2] = (k & 1) ? rank2[k / 2] | (r << 16) : r;
    __syncwarp();
    if (valid && (peers & lt_mask) == 0) s_cnt[warp][d] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  uint32_t val[VALS ? ITEMS : 1];  // loaded here: in flight over the sums and the publication
  if constexpr (VALS) {
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) val[k] = i0 + k * 32 < n ? __ldg(vals_in + i0 + k * 32) : 0u;
  }
  // digit tid: keys of the tile, published for the tiles after; places in the tile
  uint32_t cnt = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const uint32_t c = s_cnt[w][tid];
    s_cnt[w][tid] = cnt;
    cnt += c;
  }
  uint32_t* my = lookback + (size_t)tile * kRadix + tid;
  atomicExch(my, (tile == 0 ? kFlagPre : kFlagAgg) | cnt);
  const uint32_t place = cta_excl_scan(cnt, s_wsum[1]);
#pragma unroll
  for (int w = 0; w < kWarps; ++w) s_cnt[w][tid] += place;
  __syncthreads();
  // the tile in digit order
#pragma unroll
  for (int k = 0; k < ITEMS; ++k)
    if (i0 + k * 32 < n) {
      const uint32_t q = s_cnt[warp][(key[k] >> shift) & (kRadix - 1)] + ((rank2[k / 2] >> (16 * (k & 1))) & 0xffffu);
      s_key[q] = key[k];
      s_val[q] = VALS ? val[k] : (uint32_t)(i0 + k * 32);
    }
  // look back for the exclusive prefix of digit tid
  uint32_t excl = 0;
  if (tile != 0) {
    // sixteen predecessors a round trip: add their counts until one carries an
    // inclusive prefix
    constexpr int kBack = 16;
    int64_t t = (int64_t)tile - 1;
    int spins = 0;
    bool done = false;
    while (!done && t >= 0) {
      uint32_t w[kBack];
#pragma unroll
      for (int q = 0; q < kBack; ++q)
        w[q] = (t - q >= 0) ? *((const volatile uint32_t*)(lookback + (size_t)(t - q) * kRadix + tid))
                            : kFlagPre;
      int used = 0;
#pragma unroll
      for (int q = 0; q < kBack; ++q) {
        if (done || used < q) continue;  // stop at the first word not yet published
        const uint32_t v = w[q];
        if ((v & (kFlagAgg | kFlagPre)) == 0) continue;
        excl += v & kValMask;
        used = q + 1;
        if (v & kFlagPre) done = true;
      }
      t -= used;
      if (!done && used < kBack && t >= 0) {
        if (++spins > kSpinLimit) {  // give up: flag the error, treat the rest as zero
          atomicExch(err, 1u);
          break;
        }
        __nanosleep(32);
      }
    }
    atomicExch(my, kFlagPre | (excl + cnt));
  }
  s_base[tid] = dstart + excl - place;
  __syncthreads();
  const int have = (int)(n - base < kTileKeys ? n - base : kTileKeys);
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const int q = k * kSortThreads + tid;
    if (q < have) {
      const uint32_t key_q = s_key[q];
      const uint32_t pos = s_base[(key_q >> shift) & (kRadix - 1)] + (uint32_t)q;
      if (pos < n) {  // (always, but for a look-back that gave up)
        keys_out[pos] = key_q;
        vals_out[pos] = s_val[q];
      }
    }
  }
}

cudaError_t radix_sort_pairs(const uint32_t* keys_in, const uint32_t* vals_in,
                             uint32_t* keys_out, uint32_t* vals_out, uint32_t* keys_tmp,
                             uint32_t* vals_tmp, uint32_t* scratch, int64_t n, int bits,
                             cudaStream_t stream, uint32_t* epoch, const uint32_t* skip, bool clear_err) {
  if (n <= 0) return cudaSuccess;
  const int passes = passes_for(bits);
  // 2048-key tiles while they fit the SMs about once over (a tile's own chain of
  // steps is half as long), 4096-key ones beyond (half the look-back).  20-bit
  // sorts, us with 2048- / 4096-key tiles: 262,144 random pairs 41 / 52, 1,000,003
  // 74 / 65, 4,800,000 211 / 185.  (Before the warps ranked on their own, with the
  // pairs written straight from registers: 76, 100 and 304.)
  const int items = n >= (1 << 19) ? 16 : 8;
  const int ntiles = (int)((n + kSortThreads * items - 1) / (kSortThreads * items));
  uint32_t* err = sort_error_word(scratch);
  uint32_t* ghist = scratch + 256 - kMaxPasses;
  uint32_t* tile_counter = ghist + kMaxPasses * kRadix;
  uint32_t* lookback = scratch + head_words();
  // histograms, tile counters and look-back words start at zero every sort; the
  // error word before them when clear_err is set (stand-alone sorts) -- a step's
  // sort leaves it alone so it stays set until the handle reports it.
  uint32_t* from = clear_err ? scratch : ghist;
  cudaError_t e = cudaMemsetAsync(from, 0, sizeof(uint32_t) * (size_t)(lookback - from + (int64_t)passes * kRadix * ntiles),
                                  stream);
  if (e != cudaSuccess) return e;
  const int64_t hchunks = (n + kSortThreads * kHistPerThread - 1) / (kSortThreads * kHistPerThread);
  const int hist_blocks = (int)(hchunks < 608 ? hchunks : 608);
  e = launch_pdl(sort_hist_all, dim3(hist_blocks), dim3(kSortThreads), 0, stream, keys_in, n, passes, ghist, skip);
  if (e != cudaSuccess) return e;
  const uint32_t* kin = keys_in;
  const uint32_t* vin = vals_in;
  for (int p = 0; p < passes; ++p) {
    const bool to_out = ((passes - 1 - p) % 2) == 0;  // the last pass lands in keys_out
    uint32_t* ko = to_out ? keys_out : keys_tmp;
    uint32_t* vo = to_out ? vals_out : vals_tmp;
    e = launch_pdl(items == 16 ? (vin ? sort_pass<16, true> : sort_pass<16, false>)
                               : (vin ? sort_pass<8, true> : sort_pass<8, false>),
                   dim3(ntiles), dim3(kSortThreads), 0, stream, kin, vin, ko,
                   vo, n, p, (const uint32_t*)ghist, tile_counter, lookback + (size_t)p * kRadix * ntiles, err,
                   p == 0 ? epoch : (uint32_t*)nullptr, skip);
    if (e != cudaSuccess) return e;
    kin = ko;
    vin = vo;
  }
  return cudaGetLastError();
}

uint32_t* sort_error_word(uint32_t* scratch) { return scratch; }

}  // namespace sphg
