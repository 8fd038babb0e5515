// Key lengths of a right-padded batch from its boolean mask (True = keep), the form in which the attention kernels take
// the reference's key_padding_mask (training/llama/llama/models/attentions/base.py:88-103).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "sm100_ptx.cuh"

namespace hk {

// grid = B, block = 256. lens[b] = number of kept keys of row b; *bad (zero on entry) is raised by a row that does not
// keep a prefix, or keeps nothing. One launch in place of the sum / compare / reduce chain of nine that tensor
// operations need for it; a row is N bytes, so this is launch latency (about 3 us) and nothing else.
__global__ void __launch_bounds__(256) key_padding_lens_kernel(const unsigned char* mask, int32_t* lens, int32_t* bad,
                                                               int N) {
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  const unsigned char* row = mask + static_cast<size_t>(blockIdx.x) * N;
  int kept = 0, end = 0;  // kept keys, and one past the last of them
  for (int i = threadIdx.x; i < N; i += 256) {
    if (row[i]) {
      ++kept;
      end = i + 1;
    }
  }
  kept = __reduce_add_sync(0xffffffffu, kept);
  end = __reduce_max_sync(0xffffffffu, end);
  __shared__ int s_kept[8], s_end[8];
  if ((threadIdx.x & 31) == 0) {
    s_kept[threadIdx.x >> 5] = kept;
    s_end[threadIdx.x >> 5] = end;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      kept += s_kept[w];
      end = max(end, s_end[w]);
    }
    lens[blockIdx.x] = kept;
    if (kept != end || kept < 1) *bad = 1;  // every writer stores the same value
  }
}

}  // namespace hk
