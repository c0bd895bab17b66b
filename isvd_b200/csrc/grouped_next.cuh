// Work items of a grouped launch, handed out one at a time: with products of very different sizes a fixed
// stride leaves most CTAs idle while a few finish (64 uneven matrices: 1.4 ms for the 15 GFLOP of A'Q).
#pragma once

#include <cuda_runtime.h>

namespace isvdb {

// w[0] counts the items handed out beyond the first gridDim.x, w[1] the CTAs that are done; the last of
// them sets both back to zero for the next launch (launches that share w follow one another in a stream).
struct GroupedNext {
  int *w, *slot;
  int mine = 0;
  __device__ GroupedNext(int *words, int *shared) : w(words), slot(shared) {}
  __device__ void fetch() {  // the next item's number, while the current one is computed
    if (threadIdx.x == 0) mine = (int)gridDim.x + atomicAdd(w, 1);
  }
  __device__ int take() {
    __syncthreads();  // the slot's last value has been read
    if (threadIdx.x == 0) *slot = mine;
    __syncthreads();
    return *slot;
  }
  // thread 0 of every CTA, after its last item
  __device__ void done() {
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(w + 1, 1) == (int)gridDim.x - 1) {
      w[0] = 0;
      w[1] = 0;
    }
  }
};

}  // namespace isvdb
