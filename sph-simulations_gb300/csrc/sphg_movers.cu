// sphg_movers.cu -- incremental re-sort of a nearly sorted state.
//
// Between two main-loop iterations a particle moves a small fraction of a
// cell, so almost every particle keeps its cell key.  The stable sort of the
// new keys (GenericNeighborSearch::SortParticleIds,
// core/alg/GenericNeighborSearch.h:69-76, with ties in previous-slot order)
// is then a merge of two sequences:
//   * stayers: slots whose key did not change -- already in (key, slot) order,
//     because the current state is sorted;
//   * movers: slots whose key changed -- few.
// The force pass finds each mover's insertion point p while the current cell
// ranges are at hand -- the number of current slots ordered before its (new
// key, slot) -- and records it there (record_movers): a count per p, the chain
// of the movers at p, and the net change (insertions - movers) of every 512
// slots and of every 32,768.  The sorted order is then: for p = 0, 1, ..., n
// the movers of p by (key, slot), then slot p if it stays.
//
// One kernel writes it.  A block takes 512 slots with the movers inserted
// before them, whose output is one contiguous run that starts at the block's
// first slot plus the net change of the slots before it; the positions inside
// are bit counts.  Having the run's keys in shared memory, the block writes the
// cell ranges too (the keys either side of the run come from the neighbouring
// slots), so an iteration that merges needs no pass over the sorted keys.  The
// cost does not depend on how many slots changed.  When more did than
// mover_limit(), or a group or a block passed its cap, the kernel only records
// that and the full radix sort and the reorder run instead (under a conditional
// graph node, or they return at once on the decision word).
#include <cstdint>

#include <cuda_runtime.h>

#include "sphg_common.cuh"
#include "sphg_movers.cuh"
#include "sphg_movers_body.cuh"

namespace sphg {

namespace {

__global__ void __launch_bounds__(kMergeThreads) movers_merge(MoverArgs a) {
  __shared__ MergeShared sh;
  cudaGridDependencySynchronize();  // the mover record of the previous force pass
  allow_next_kernel(a.early_next);
  merge_block<kKernels>(a, sh, blockIdx.x, *(volatile const uint32_t*)a.rec.next_epoch);
}

}  // namespace

cudaError_t launch_movers(const MoverArgs& a, cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  // the block of p = n included
  cudaError_t e = launch_pdl(movers_merge, dim3((unsigned)((a.n >> kMergeShift) + 1)), dim3(kMergeThreads), 0, st, a);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

}  // namespace sphg
