// Span-kernel instantiations of the exact-sampling costs, 16 warps: SAD_AVG, SQD_REF and NCC_REF with 4
// points per warp (one channel: tiles of 256 columns, three: 64, whose windows have three planes) and
// three-channel MI with 2; plain and self-checking.
#include "cgs_internal.h"
#include "cgs_span_exact.cuh"

namespace cgs {

template <int COST, int G, int TX1>
static const void *exact16(int C, int TX, bool check) {
    if (C == 1 && TX == TX1)
        return check ? (const void *)span_exact_kernel<COST, 1, G, 16, TX1, true>
                     : (const void *)span_exact_kernel<COST, 1, G, 16, TX1, false>;
    if (C == 3 && TX == 2)
        return check ? (const void *)span_exact_kernel<COST, 3, G, 16, 2, true>
                     : (const void *)span_exact_kernel<COST, 3, G, 16, 2, false>;
    return nullptr;
}

const void *kernel_span_exact(int cost, int C, int G, int TX, bool check) {
    switch (cost) {
        case CGS_COST_SAD_AVG: return G == 4 ? exact16<CGS_COST_SAD_AVG, 4, 8>(C, TX, check) : nullptr;
        case CGS_COST_SQD_REF: return G == 4 ? exact16<CGS_COST_SQD_REF, 4, 8>(C, TX, check) : nullptr;
        case CGS_COST_NCC_REF: return G == 4 ? exact16<CGS_COST_NCC_REF, 4, 8>(C, TX, check) : nullptr;
        case CGS_COST_MI:
            if (G != 2 || C != 3 || TX != 2) return nullptr;
            return check ? (const void *)span_exact_kernel<CGS_COST_MI, 3, 2, 16, 2, true>
                         : (const void *)span_exact_kernel<CGS_COST_MI, 3, 2, 16, 2, false>;
        default: return nullptr;
    }
}

size_t span_kernel_smem(int G, int NW, int TH, int TX, int tiles, int cap, bool exact, int mi_bins) {
    return span_smem_bytes(G, NW, TH, TX, tiles, cap) + (exact ? span_exact_extra(G, NW, TH, mi_bins) : 0);
}

}  // namespace cgs
