// Span-kernel instantiations of the exact-sampling costs (SAD_AVG, SQD_REF, NCC_REF), 16 warps of 4
// points: one channel with tiles of 256 columns, three with tiles of 64 (three planes of windows in
// the stage); plain and, for one channel, self-checking.
#include "cgs_internal.h"
#include "cgs_span_exact.cuh"

namespace cgs {

template <int COST>
static const void *exact16(int C, int TX, bool check) {
    if (C == 1 && TX == 8)
        return check ? (const void *)span_exact_kernel<COST, 1, 4, 16, 8, true>
                     : (const void *)span_exact_kernel<COST, 1, 4, 16, 8, false>;
    if (C == 3 && TX == 2 && !check) return (const void *)span_exact_kernel<COST, 3, 4, 16, 2, false>;
    return nullptr;
}

const void *kernel_span_exact(int cost, int C, int TX, bool check) {
    switch (cost) {
        case CGS_COST_SAD_AVG: return exact16<CGS_COST_SAD_AVG>(C, TX, check);
        case CGS_COST_SQD_REF: return exact16<CGS_COST_SQD_REF>(C, TX, check);
        case CGS_COST_NCC_REF: return exact16<CGS_COST_NCC_REF>(C, TX, check);
        default: return nullptr;
    }
}

}  // namespace cgs
