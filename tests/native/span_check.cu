// Device functions of the span kernels by themselves: span_check CASE prints the words that
// tests/test_span_device_gpu.py compares.
//   bounds     status after a part that found a bad address and was not its task's last one
//   lost       a part after one that a CTA that gave up did not run, and that order turned around:
//              what join_parts returned, tasks done, status, whether the argmin key is untouched
//   quotients  exact_quot2 against IEEE division: quotients tried, quotients that differ, over mantissas near
//              the binade's ends, near multiples of each other and random ones, exponents over quot_range's
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

// 24-bit mantissa i of kind k: the binade's ends, few bits set, all but few, or mixed from a counter.
__device__ uint32_t mantissa(uint32_t i, uint32_t k) {
    const uint32_t h = (i * 2654435761u) ^ ((i * 0x9e3779b9u) >> 15), r = h ^ (h >> 13) ^ (h << 7);
    const uint32_t j = i % 23u, l = (i / 23u) % 23u;
    if (k == 0u) return i % 64u;                            // 1 + a few ulps
    if (k == 1u) return 0x7fffffu - i % 64u;                // 2 - a few ulps
    if (k == 2u) return (1u << j | 1u << l) & 0x7fffffu;    // few bits
    if (k == 3u) return ~(1u << j | 1u << l) & 0x7fffffu;   // all but few
    return r & 0x7fffffu;
}

// Quotients X / w of mantissas of kinds (kx, kw), n per thread, signs and exponents mixed: |w| in
// [2^-40, 2^40], |X| in [2^-93, 2^60] or 0, and results in the normal range, as the callers' are.
__global__ void quotient_kernel(uint32_t kx, uint32_t kw, uint32_t n, unsigned long long *tried, unsigned long long *wrong) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long t = 0, bad = 0;
    auto same = [](float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a == 0.0f && b == 0.0f); };
    for (uint32_t i = 0; i < n; i++) {
        const uint32_t c = tid * n + i, e = c * 747796405u + 2891336453u;
        const int ew = (int)((e >> 8) % 81u) - 40, ex = (int)((e >> 16) % 140u) - 80;
        const float w = __uint_as_float((uint32_t)(ew + 127) << 23 | mantissa(c, kw)) * (e & 1u ? -1.0f : 1.0f);
        float X = __uint_as_float((uint32_t)(ex + 127) << 23 | mantissa(c / 7u, kx)) * (e & 2u ? -1.0f : 1.0f);
        const float Y = __uint_as_float((uint32_t)(ew / 2 + 127) << 23 | mantissa(c ^ 0x5bd1u, kx));
        if (e % 1021u == 0u) X = 0.0f;
        float2 x, y;
        exact_quot2(make_float2(w, -w), make_float2(-X, X), make_float2(-Y, Y), x, y);
        t += 4;
        bad += !same(x.x, __fdiv_rn(X, w)) + !same(x.y, __fdiv_rn(-X, -w)) + !same(y.x, __fdiv_rn(Y, w)) +
               !same(y.y, __fdiv_rn(-Y, -w));
    }
    atomicAdd(tried, t);
    atomicAdd(wrong, bad);
}

static void quotients() {
    unsigned long long *tried = zeroed<unsigned long long>(1), *wrong = zeroed<unsigned long long>(1);
    for (uint32_t kx = 0; kx < 5; kx++)
        for (uint32_t kw = 0; kw < 5; kw++) quotient_kernel<<<592, 256>>>(kx, kw, 256, tried, wrong);
    check(cudaGetLastError());
    check(cudaDeviceSynchronize());
    std::printf("%llu %llu\n", value(tried), value(wrong));
}

int main(int argc, char **argv) {
    const std::string c = argc > 1 ? argv[1] : "";
    if (c == "bounds") bounds();
    else if (c == "lost") lost();
    else if (c == "quotients") quotients();
    else return 1;
    return 0;
}
