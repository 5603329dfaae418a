// Host check of the index a warp of bulk_runs_kernel takes, at run counts no
// test can allocate: the 32-bit thread number wraps from 2^27 runs on.
#include <cstdio>

#include "bfvm_kernels.cuh"

int main() {
  for (int64_t run : {INT64_C(0), INT64_C(7), INT64_C(8), (INT64_C(1) << 27) - 1, INT64_C(1) << 27,
                      (INT64_C(1) << 27) + 5, (INT64_C(1) << 31) - 1})
    for (uint32_t lane : {0u, 31u}) {
      const uint32_t block = (uint32_t)(run / 8), thread = (uint32_t)(run % 8) * 32 + lane;
      if (bfvm::bulk_run(block, thread) != run) {
        std::printf("run %lld: block %u thread %u gives %lld\n", (long long)run, block, thread,
                    (long long)bfvm::bulk_run(block, thread));
        return 1;
      }
    }
  return 0;
}
