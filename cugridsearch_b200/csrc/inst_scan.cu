// Kernel instantiations of the scanline functors calcSQDAlt, calcNCCAlt and calcMIAlt.
#include "cgs_internal.h"
#include "cgs_scan.cuh"

namespace cgs {

const void *kernel_scan(int cost, int C) {
    if (C == 1) {
        if (cost == CGS_COST_SQD_ALT) return (const void *)scan_sum_kernel<CGS_COST_SQD_ALT, 1>;
        if (cost == CGS_COST_NCC_ALT) return (const void *)scan_sum_kernel<CGS_COST_NCC_ALT, 1>;
        if (cost == CGS_COST_MI_ALT) return (const void *)scan_kernel<1>;
    } else if (C == 3) {
        if (cost == CGS_COST_SQD_ALT) return (const void *)scan_sum_kernel<CGS_COST_SQD_ALT, 3>;
        if (cost == CGS_COST_NCC_ALT) return (const void *)scan_sum_kernel<CGS_COST_NCC_ALT, 3>;
        if (cost == CGS_COST_MI_ALT) return (const void *)scan_kernel<3>;
    }
    return nullptr;
}

size_t scan_smem_bytes(int cost) {
    if (cost != CGS_COST_MI_ALT) return 0;  // scan_sum_kernel's is static
    return 8 * kScanWarps + (size_t)kScanWarps * kScanRows * (sizeof(RowInfo) + kMaxSegs * sizeof(Seg)) +
           (size_t)kScanWarps * 65 * 65 * 4;
}

}  // namespace cgs
