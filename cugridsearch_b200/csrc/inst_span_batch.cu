// The multi-pair span kernel of batches: 16 warps of 4 points, tiles of 256 columns.
#include "cgs_internal.h"
#include "cgs_span_batch.cuh"

namespace cgs {

const void *kernel_span_batch(int G, int NW, int TX, bool zncc, bool check) {
    if (G != 4 || NW != 16 || TX != 8 || check) return nullptr;
    return zncc ? (const void *)span_batch_kernel<4, 16, 8, true, false>
                : (const void *)span_batch_kernel<4, 16, 8, false, false>;
}

}  // namespace cgs
