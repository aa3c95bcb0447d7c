// mrsph_sort.cu — the per-handle kernels of the cell binning's counting sort
// (block functions in mrsph_sort.cuh).
#include <cuda_runtime.h>

#include "engine_iface.h"
#include "mrsph_sort.cuh"

namespace mrsph {

namespace {
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const int* __restrict__ counts, long long n,
                                                             int* __restrict__ blocksums) {
  chain_wait();
  scan_reduce_block(counts, n, blocksums, blockIdx.x);
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_top(int* blocksums, int nb) {
  chain_wait();
  scan_top_block(blocksums, nb);
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_down(int* __restrict__ counts, long long n,
                                                           const int* __restrict__ blocksums,
                                                           int* __restrict__ cstart, int ntotal, int from) {
  chain_wait();
  scan_down_block(counts, n, blocksums, cstart, ntotal, blockIdx.x, from);
}

__global__ void k_scatter(const int* __restrict__ cellkey, const int* __restrict__ id, int* cursor,
                          const int* __restrict__ cstart, int* __restrict__ perm, int* __restrict__ pid, long long n) {
  chain_wait();
  scatter_block(cellkey, id, cursor, cstart, perm, pid, n, blockIdx.x);
}
}  // namespace

// block totals of the smallest chunk (the batch kernels' 256-thread scans)
long long scan_blocksums_size(long long ncells) { return (ncells + SCAN_CHUNK_MIN - 1) / SCAN_CHUNK_MIN + 1; }

// Up to this many blocks a block adds up the totals before it itself: 2048
// words from L2 at most.  (The top pass is a launch of one block; at 6,102
// blocks it takes 7.6 us, less than the blocks' own sums would.)
constexpr int kSelfPrefix = 2048;

void cell_scan(int* counts, int* cstart, int* blocksums, long long ncells, int ntotal, cudaStream_t s) {
  const int nb = (int)((ncells + SCAN_CHUNK - 1) / SCAN_CHUNK);
  if (nb > 1) launch_chained(k_scan_reduce, nb, SCAN_THREADS, s, counts, ncells, blocksums);
  if (nb > kSelfPrefix) launch_chained(k_scan_top, 1, SCAN_THREADS, s, blocksums, nb);
  launch_chained(k_scan_down, nb, SCAN_THREADS, s, counts, ncells, blocksums, cstart, ntotal,
                 nb == 1 ? (int)SCAN_SINGLE : nb > kSelfPrefix ? (int)SCAN_PREFIX : (int)SCAN_TOTALS);
}

void cell_scatter(const int* cellkey, const int* id, int* cursor, const int* cstart, int* perm, int* pid, long long n,
                  cudaStream_t s) {
  const int nb = (int)((n + 255) / 256);
  launch_chained(k_scatter, nb, 256, s, cellkey, id, cursor, cstart, perm, pid, n);
}

}  // namespace mrsph
