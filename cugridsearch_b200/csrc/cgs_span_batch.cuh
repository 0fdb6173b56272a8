// cgs_span_batch.cuh -- the multi-pair span kernel.
//
// Batches: the tasks of many single-channel pairs of the span costs (zero-mean NCC on fast samples,
// SAD_AVG, SQD_REF and NCC_REF on exact ones; each pair with its own staged planes, prefix sums,
// tiles and grid) from one counter, so that pairs too small to fill the GPU alone share it and one
// cost's last tasks overlap the next cost's first.  A task's pair is found in the prefix of task
// counts; its parameters are read from global memory and its cost selects the task body.  Shared
// memory is carved once for the largest tile count of the pairs and one window stage size (`cap`)
// for all of them; each pair's results are those of its single-pair kernel.
#pragma once
#include "cgs_span_exact.cuh"

namespace cgs {

// One task of a pair, by the pair's cost.  ZNCC: every pair's (the proposal serving's levels): a kernel of
// their body alone, 3 % faster than beside the others' in one register allocation.
template <int G, int NW, int TX, bool ZNCC, bool CHECK>
__device__ __forceinline__ bool run_pair_task(const SearchParams &p, uint32_t task, const SpanSmem &ss, uint32_t &wit) {
    if constexpr (ZNCC) return run_span_task<G, NW, TX, CHECK>(p, task, ss, wit);
    switch (p.cost) {
        case CGS_COST_SAD_AVG: return run_span_exact_task<CGS_COST_SAD_AVG, 1, G, NW, TX, CHECK, true>(p, task, ss, wit);
        case CGS_COST_SQD_REF: return run_span_exact_task<CGS_COST_SQD_REF, 1, G, NW, TX, CHECK, true>(p, task, ss, wit);
        case CGS_COST_NCC_REF: return run_span_exact_task<CGS_COST_NCC_REF, 1, G, NW, TX, CHECK, true>(p, task, ss, wit);
        default: return run_span_task<G, NW, TX, CHECK>(p, task, ss, wit);
    }
}

template <int G, int NW, int TX, bool ZNCC, bool CHECK>
__global__ void __launch_bounds__(NW * 32, 1) span_batch_kernel(const __grid_constant__ SpanBatchParams b) {
    extern __shared__ __align__(128) unsigned char smem[];
    const SpanSmem ss = carve_span<G, NW>(smem, b.tile_h, TX, b.tiles, b.cap, true);
    // the task word sits in the carve's head, after the flags (no static shared memory: the
    // dynamic carve may take all 227 KB)
    volatile uint32_t &s_task = *reinterpret_cast<volatile uint32_t *>(ss.bounds_flag + 1);
    if (threadIdx.x == 0) {
        mbar_init(ss.bar, 1);
        fence_mbar_init();
        *ss.abort_flag = 0;
        *ss.bounds_flag = 0;
    }
    uint32_t wit = 0;
    for (;;) {
        __syncthreads();  // the previous task is done with s_task
        if (threadIdx.x == 0) s_task = atomicAdd(b.next_task, 1u);
        __syncthreads();
        const uint32_t t = s_task;
        if (t >= b.total_tasks) return;
        uint32_t lo = 0, hi = b.n_pairs;  // task_begin[lo] <= t < task_begin[hi]
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(b.task_begin + mid) <= t) lo = mid;
            else hi = mid;
        }
        const SearchParams &p = b.pairs[lo];
        const uint32_t slot = __ldg(b.slot + lo);
        if (threadIdx.x == 0 && b.t_start) atomicMin(b.t_start + slot, (unsigned long long)global_ns());
        if (!run_pair_task<G, NW, TX, ZNCC, CHECK>(p, t - __ldg(b.task_begin + lo), ss, wit)) {
            if (threadIdx.x == 0) {
                // retire this task and every task not yet taken, with the timeout status
                retire_tasks(p, ~0ull, 1u, true);
                for (;;) {
                    const uint32_t u = atomicAdd(b.next_task, 1u);
                    if (u >= b.total_tasks) break;
                    uint32_t l2 = 0, h2 = b.n_pairs;
                    while (h2 - l2 > 1) {
                        const uint32_t mid = (l2 + h2) >> 1;
                        if (__ldg(b.task_begin + mid) <= u) l2 = mid;
                        else h2 = mid;
                    }
                    retire_tasks(b.pairs[l2], ~0ull, 1u, true);
                }
            }
            return;
        }
        if (threadIdx.x == 0 && b.t_end) atomicMax(b.t_end + slot, (unsigned long long)global_ns());
    }
}

}  // namespace cgs
