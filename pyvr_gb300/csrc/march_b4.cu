// Batch march kernel instantiated for 4^3-texel bricks (see march_core.cuh).
#include "march_core.cuh"

namespace pvr {

const void *batch_kernel_b2(const Tuning &t, int variant) { return batch_kernel_log2<2>(t, variant); }

const void *split_kernel_b2(int lanes, int variant) { return split_kernel_log2<2>(lanes, variant); }

const void *single_kernel_b2(const Tuning &t, int variant) { return single_kernel_log2<2>(t, variant); }

int max_batch_blocks_b2(const Tuning &t, int lut_smem_entries, int variant) {
    return max_blocks_log2<2>(t, lut_smem_entries, variant);
}

}  // namespace pvr
