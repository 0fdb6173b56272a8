// Device functions of the span kernels by themselves: span_check CASE prints the words that
// tests/test_span_device_gpu.py compares.
//   bounds     status after a part that found a bad address and was not its task's last one
//   lost       a part after one that a CTA that gave up did not run, and that order turned around:
//              what join_parts returned, tasks done, status, whether the argmin key is untouched
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>

#include "cgs_internal.h"
#include "cgs_span.cuh"

using namespace cgs;

constexpr int G = 4, NW = 16, TH = 16, TX = 8, TILES = 2, CAP = 4096;

static void check(cudaError_t e) {
    if (e == cudaSuccess) return;
    std::fprintf(stderr, "%s\n", cudaGetErrorString(e));
    std::exit(2);
}

template <class T>
static T *zeroed(size_t n) {
    T *p;
    check(cudaMalloc(&p, n * sizeof(T)));
    check(cudaMemset(p, 0, n * sizeof(T)));
    return p;
}

template <class T>
static T value(const T *p) {
    T v;
    check(cudaMemcpy(&v, p, sizeof(T), cudaMemcpyDeviceToHost));
    return v;
}

// One task of two bands, split into two parts.
static SearchParams two_parts() {
    SearchParams p;
    std::memset(&p, 0, sizeof(p));
    p.dims = 8;
    p.n = G * NW;
    p.num_tasks = 1;
    p.splits = 2;
    p.tiles_x = 1;
    p.tiles_y = TILES;
    p.tile_h = TH;
    p.key = zeroed<unsigned long long>(1);
    check(cudaMemset(p.key, 0xff, 8));
    p.done = zeroed<unsigned int>(1);
    p.status = zeroed<unsigned int>(1);
    p.result = zeroed<cgs_argmin>(1);
    p.split_tot = zeroed<double>((size_t)TILES * NW * G * 5);
    p.split_cnt = zeroed<int>(2 * NW * G);
    p.split_done = zeroed<unsigned int>(1);
    return p;
}

// Joins part `part`, whose CTA found a bad address if `found`; out: what join_parts returned.
__global__ void __launch_bounds__(NW * 32, 1) join_kernel(const __grid_constant__ SearchParams p, int part, int found, int *out) {
    extern __shared__ __align__(128) unsigned char smem[];
    const SpanSmem ss = carve_span<G, NW>(smem, TH, TX, TILES, CAP);
    if (threadIdx.x == 0) *ss.bounds_flag = found;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = lane; i < G * 5; i += 32) ss.dtot[warp * G * 5 + i] = 0.0;
    if (lane < G) ss.cnt[warp * G + lane] = 1;
    __syncthreads();
    const bool last = join_parts<G, NW, true>(p, 0, part, ss, ss.dtot + warp * G * 5, ss.cnt + warp * G);
    if (threadIdx.x == 0) *out = last ? 1 : 0;
}

static int join(const SearchParams &p, int part, int found) {
    const size_t smem = span_smem_bytes(G, NW, TH, TX, TILES, CAP);
    check(cudaFuncSetAttribute(join_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int *out = zeroed<int>(1);
    join_kernel<<<1, NW * 32, smem>>>(p, part, found, out);
    check(cudaGetLastError());
    check(cudaDeviceSynchronize());
    return value(out);
}

static void bounds() {
    const SearchParams p = two_parts();
    const int first = join(p, 1, 1);
    const unsigned int after = value(p.status);
    const int last = join(p, 0, 0);
    std::printf("%d %u %d %u\n", first, after & kStatusSpanBounds, last, value(p.status) & kStatusSpanBounds);
}

// What a CTA that gives up on part `part` does.
__global__ void lose_kernel(const __grid_constant__ SearchParams p, int part) { retire_parts(p, (uint32_t)part, 2u, 2u); }

static void lost() {
    for (int first = 0; first < 2; first++) {
        const SearchParams p = two_parts();
        int joined = 0;
        if (first == 1) joined = join(p, 1, 0);
        lose_kernel<<<1, 1>>>(p, 0);
        check(cudaGetLastError());
        check(cudaDeviceSynchronize());
        if (first == 0) joined = join(p, 1, 0);
        std::printf("%d %u %u %d\n", joined, value(p.done), value(p.status), value(p.key) == ~0ull);
    }
}

int main(int argc, char **argv) {
    const std::string c = argc > 1 ? argv[1] : "";
    if (c == "bounds") bounds();
    else if (c == "lost") lost();
    else return 1;
    return 0;
}
