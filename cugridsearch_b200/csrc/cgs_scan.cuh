// cgs_scan.cuh -- the scanline functors calcNCCAlt, calcSQDAlt and calcMIAlt on sm_100a.
//
// These reference functors (src/gpu/cudaErrorFunctions.cuh:226-376,
// src/gpu/cudaErrorFunction_mi.cuh:117-255) do not loop over fixed pixels: for each fixed row
// they intersect the row's image under the homography with the moving image
// (parametricAssignValues[Norm], cudaImageFunctions.cuh:315-441), then step a float lambda
// along the row by repeated addition, sampling the moving image at lambda * v + p0 and the
// fixed image at (row, lambda).  Which samples exist, where they lie and the overlap gates
// all follow float recurrences; cgs_seq.cuh reproduces those recurrences exactly, so each
// lane can jump straight to its own lambda.
//
// Work layout: one warp per grid point (persistent over grid points in the locality order of
// the pixel kernel).  For each block of 32 rows every lane sets up one row (the exact
// intersection, ~100 correctly rounded operations), the warp then walks the rows, lanes
// taking every 32nd lambda.  calcMIAlt (scan_kernel) reads both images through L1 from the staged
// planes, whose extra column and zero row make the reference's flat-index neighbours explicit;
// calcNCCAlt and calcSQDAlt (scan_sum_kernel) read tap quads and pairs made from them.
#pragma once
#include "cgs_kernels.cuh"
#include "cgs_seq.cuh"

namespace cgs {

// parametersToHomographyNorm (src/gpu/cudaImageFunctions.cuh:181-214): integer size ratios,
// rounded integer centres (cmy from the moving WIDTH, :201), scale divided by the ratios.
__device__ __forceinline__ Homog h_norm(const float *q, float c, float s, int mw, int mh, int fw, int fh) {
    const float x_ratio = (float)(fw / mw), y_ratio = (float)(fh / mh);
    const float cfx = (float)(fw / 2), cfy = (float)(fh / 2), cmx = (float)(mw / 2), cmy = (float)(mw / 2);
    const float sx = xd(q[1], x_ratio), sy = xd(q[2], y_ratio), sh = q[3], tx = q[4], ty = q[5];
    Homog h;
    h.h11 = xm(sx, c);
    h.h12 = xs(xm(xm(sy, sh), c), xm(sy, s));
    h.h13 = xd(xa(xs(tx, cfx), cmx), (float)fw);
    h.h21 = xm(sx, s);
    h.h22 = xa(xm(xm(sy, sh), s), xm(sy, c));
    h.h23 = xd(xa(xs(ty, cfy), cmy), (float)fh);
    h.h31 = q[6];
    h.h32 = q[7];
    return h;
}

struct RowInfo {
    float ls, le;        // first lambda, exclusive lambda limit (min of the reference's two bounds)
    float vx, vy, p0x, p0y;
    float rowv;          // fixed-image row coordinate of the samples
    uint32_t n;          // number of lambda samples (0 when the row misses the moving image)
    int nseg;            // lambda segments; -1: more than kMaxSegs (lanes step explicitly)
};

constexpr int kMaxSegs = 24;

// parametricAssignValues (cudaImageFunctions.cuh:315-376) in the reference's operation order.
__device__ inline void assign_values(const Homog &H, int m_width, int m_height, int f_width, int f_height, int row_i,
                                     float &ls, float &le, float &v_x, float &v_y, float &p0_x, float &p0_y,
                                     bool &in) {
    const float h11 = H.h11, h12 = H.h12, h13 = H.h13, h21 = H.h21, h22 = H.h22, h23 = H.h23, h31 = H.h31,
                h32 = H.h32;
    const float row = (float)row_i, fw = (float)f_width, mh = (float)m_height, mw = (float)m_width;
    const float D = xs(xa(xa(xs(xs(xm(h11, h22), xm(h12, h21)), xm(xm(h11, h23), h32)), xm(xm(h12, h23), h31)),
                          xm(xm(h13, h21), h32)),
                       xm(xm(h13, h22), h31));
    const float den1 = xa(xs(xs(xm(h11, h22), xm(h12, h21)), xm(xm(h11, h32), row)), xm(xm(h12, h31), row));
    const float den2 = xa(xs(xs(xa(xs(xm(h11, h22), xm(h12, h21)), xm(xm(fw, h21), h32)), xm(xm(fw, h22), h31)),
                             xm(xm(h11, h32), row)),
                          xm(xm(h12, h31), row));
    const float dd = xm(den1, den2);
    v_x = xd(xm(xs(h22, xm(h32, row)), D), dd);
    v_y = xd(-xm(xs(h21, xm(h31, row)), D), dd);
    const float pden = xa(xs(xm(h12, h21), xm(h11, h22)), xm(row, xs(xm(h11, h32), xm(h12, h31))));
    p0_x = xd(xa(xs(xm(h13, h22), xm(h12, h23)), xm(row, xs(h12, xm(h13, h32)))), pden);
    p0_y = xd(-xa(xs(xm(h13, h21), xm(h11, h23)), xm(row, xs(h11, xm(h13, h31)))), pden);
    const float a21 = xs(h21, xm(h31, row)), a22 = xs(h22, xm(h32, row));
    const float inner1 = xa(xs(xs(xm(h11, h23), xm(h13, h21)), xm(h11, row)), xm(xm(h13, h31), row));
    const float lambda_top = xd(-xm(inner1, den2), xm(a21, D));
    const float x_top_ipt = xd(-xs(h23, row), a21);
    const float inner2 =
        xa(xs(xa(xs(xa(xs(xs(xm(h11, h23), xm(h13, h21)), xm(h11, row)), xm(xm(h11, h22), mh)), xm(xm(h12, h21), mh)),
                 xm(xm(h13, h31), row)),
              xm(xm(xm(h11, h32), mh), row)),
           xm(xm(xm(h12, h31), mh), row));
    const float lambda_bottom = xd(-xm(den2, inner2), xm(a21, D));
    const float x_bottom_ipt = xd(-xs(xa(xs(h23, row), xm(h22, mh)), xm(xm(h32, mh), row)), a21);
    const float inner3 = xa(xs(xs(xm(h12, h23), xm(h13, h22)), xm(h12, row)), xm(xm(h13, h32), row));
    const float lambda_left = xd(-xm(inner3, den2), xm(a22, D));
    const float y_left_ipt = xd(-xs(h23, row), a22);
    const float inner4 =
        xs(xa(xa(xa(xs(xs(xs(xm(h12, h23), xm(h13, h22)), xm(h12, row)), xm(xm(h11, h22), mw)), xm(xm(h12, h21), mw)),
                 xm(xm(h13, h32), row)),
              xm(xm(xm(h11, h32), mw), row)),
           xm(xm(xm(h12, h31), mw), row));
    const float lambda_right = xd(-xm(den2, inner4), xm(a22, D));
    const float y_right_ipt = xd(-xs(xa(xs(h23, row), xm(h21, mw)), xm(xm(h31, mw), row)), a22);
    if (x_top_ipt >= 0 && x_top_ipt < m_width && lambda_top >= 0 && lambda_top < f_width) {
        if (v_y > 0) ls = lambda_top; else le = lambda_top;
        in = true;
    }
    if (x_bottom_ipt >= 0 && x_bottom_ipt < m_width && lambda_bottom >= 0 && lambda_bottom < f_width) {
        if (v_y < 0) ls = lambda_bottom; else le = lambda_bottom;
        in = true;
    }
    if (y_left_ipt >= 0 && y_left_ipt < m_height && lambda_left >= 0 && lambda_left < f_height) {
        if (v_x > 0) ls = lambda_left; else le = lambda_left;
        in = true;
    }
    if (y_right_ipt >= 0 && y_right_ipt < m_height && lambda_right >= 0 && lambda_right < f_height) {
        if (v_x < 0) ls = lambda_right; else le = lambda_right;
        in = true;
    }
}

// parametricAssignValuesNorm (cudaImageFunctions.cuh:378-441) in the reference's order.
__device__ inline void assign_values_norm(const Homog &H, float row, float &ls, float &le, float &v_x, float &v_y,
                                          float &p0_x, float &p0_y, bool &in) {
    const float h11 = H.h11, h12 = H.h12, h13 = H.h13, h21 = H.h21, h22 = H.h22, h23 = H.h23, h31 = H.h31,
                h32 = H.h32;
    const float col = -0.5f;
    const float D = xs(xa(xa(xs(xs(xm(h11, h22), xm(h12, h21)), xm(xm(h11, h23), h32)), xm(xm(h12, h23), h31)),
                          xm(xm(h13, h21), h32)),
                       xm(xm(h13, h22), h31));
    const float a21 = xs(h21, xm(h31, row)), a22 = xs(h22, xm(h32, row));
    v_y = xd(-a21, D);
    v_x = xd(a22, D);
    const float den = xs(xa(xs(xm(h11, h22), xm(h12, h21)), xm(col, xs(xm(h21, h32), xm(h22, h31)))),
                         xm(row, xs(xm(h11, h32), xm(h12, h31))));
    const float numx = xs(xa(xs(xm(h12, h23), xm(h13, h22)), xm(col, xs(h22, xm(h23, h32)))),
                          xm(row, xs(h12, xm(h13, h32))));
    const float numy = xs(xa(xs(xm(h11, h23), xm(h13, h21)), xm(col, xs(h21, xm(h23, h31)))),
                          xm(row, xs(h11, xm(h13, h31))));
    p0_x = xd(numx, den);
    p0_y = xd(-numy, den);
    const float qy = xd(numy, den), qx = xd(numx, den);
    const float two_h23 = xm(2.0f, h23), two_row = xm(2.0f, row);
    const float lambda_top = xd(-xm(xs(qy, 0.5f), D), a21);
    const float x_top_ipt = xd(xs(xa(xs(h22, two_h23), two_row), xm(h32, row)), xm(2.0f, a21));
    const float lambda_bottom = xd(-xm(xa(qy, 0.5f), D), a21);
    const float x_bottom_ipt = xd(-xs(xs(xa(h22, two_h23), two_row), xm(h32, row)), xm(2.0f, a21));
    const float lambda_left = xd(-xm(xa(qx, 0.5f), D), a22);
    const float y_left_ipt = xd(xs(xa(xs(h21, two_h23), two_row), xm(h31, row)), xm(2.0f, a22));
    const float lambda_right = xd(-xm(xs(qx, 0.5f), D), a22);
    const float y_right_ipt = xd(-xs(xs(xa(h21, two_h23), two_row), xm(h31, row)), xm(2.0f, a22));
    if (x_top_ipt > -0.5f && x_top_ipt < 0.5f && lambda_top >= 0 && lambda_top < 1) {
        if (v_y > 0) ls = lambda_top; else le = lambda_top;
        in = true;
    }
    if (x_bottom_ipt > -0.5f && x_bottom_ipt < 0.5f && lambda_bottom > 0 && lambda_bottom < 1) {
        if (v_y < 0) ls = lambda_bottom; else le = lambda_bottom;
        in = true;
    }
    if (y_left_ipt > -0.5f && y_left_ipt < 0.5f && lambda_left > 0 && lambda_left < 1) {
        if (v_x > 0) ls = lambda_left; else le = lambda_left;
        in = true;
    }
    if (y_right_ipt > -0.5f && y_right_ipt < 0.5f && lambda_right > 0 && lambda_right < 1) {
        if (v_x < 0) ls = lambda_right; else le = lambda_right;
        in = true;
    }
}

// CudaImage::valueAt_bilinear including its inImage test (0 outside), reference order.
__device__ __forceinline__ float value_exact(const float *pl, int pitch, float wf, float hf, float y, float x) {
    return in_image(y, x, wf, hf) ? bilinear_in(pl, pitch, y, x) : 0.0f;
}

constexpr int kScanRows = 32;  // rows set up per block (one per lane)
constexpr int kScanWarps = 8;  // warps per CTA (one grid point each)

// The CTA's best key into the search's, and the result by the last CTA (one thread).
__device__ __forceinline__ void scan_finish(const SearchParams &p, const unsigned long long *wbest) {
    unsigned long long b = ~0ull;
    for (int w = 0; w < kScanWarps; w++) b = wbest[w] < b ? wbest[w] : b;
    if (b != ~0ull) atomicMin(p.key, b);
    __threadfence();
    const unsigned int ticket = atomicAdd(p.done, 1u);
    if (ticket == gridDim.x - 1) {
        __threadfence();
        write_result(p);
    }
}

// x_0 = x, x_1 = fl(x + 1), ... below limit, as runs of exact unit steps: seq_segments for an
// increment of 1, where every binade's ulp divides the step (0 <= x, limit < 2^23) and no run stalls.
// segs: {first index, its value's bits} per run.
constexpr int kMaxUnitSegs = 16;  // lambda up to 2^14; more runs: lanes step explicitly
__device__ __forceinline__ uint32_t unit_segments(float x, float limit, uint2 *segs, int &nseg) {
    nseg = 0;
    uint32_t k = 0;
    while (x < limit) {
        if (nseg < kMaxUnitSegs) segs[nseg] = make_uint2(k, __float_as_uint(x));
        nseg++;
        if (x >= 1.0f) {  // below 1 a step always leaves the binade
            const float end = __uint_as_float(__float_as_uint(x) | 0x7fffffu);  // the binade's last value
            const float n_in = floorf(end - x);                                 // exact: multiples of one ulp
            const double n_lim = ceil((double)limit - (double)x) - 1.0;         // exact: at most 48 bits
            if (n_lim < (double)n_in) return k + (uint32_t)n_lim + 1u;
            k += (uint32_t)n_in;
            x += n_in;
        }
        x = xa(x, 1.0f);
        k++;
    }
    return k;
}

struct SumRow {
    float vx, vy, p0x, p0y;
    float ls, mag;   // first lambda; |v| (the reference's mov_area increment)
    uint32_t n;      // number of lambda samples (0 when the row misses the moving image)
    int nseg;        // runs; above kMaxUnitSegs: lanes step explicitly
};

// One lambda sample of the sums.  The moving image comes as tap quads {v00, v10, v01 - v00, v11 - v10},
// the fixed one, sampled on a whole row where the lower taps' weight is 0, as pairs {v0, v1 - v0}: one
// load per channel and image (eight scalar ones took 36.9 warp instructions per 32 samples of a
// channel), and the same roundings as interpolating the taps.
template <int C>
struct SumSample {
    float4 m[C];
    float2 f[C];
    float ax, ay, af;
    bool inside;
    __device__ __forceinline__ void load(const SearchParams &p, const SumRow &r, float2 nzero2, float lam,
                                         uint32_t frow) {
        constexpr float kMagic = 8388608.0f;      // 2^23: rounding down onto the integers
        constexpr uint32_t kBits = 0x4b000000u;
        const float2 pos = __fadd2_rn(__ffma2_rn(make_float2(lam, lam), make_float2(r.vx, r.vy), nzero2),
                                      make_float2(r.p0x, r.p0y));
        const float tx = __fadd_rd(pos.x, kMagic), ty = __fadd_rd(pos.y, kMagic), tl = __fadd_rd(lam, kMagic);
        const uint32_t ux = __float_as_uint(tx) - kBits, uy = __float_as_uint(ty) - kBits;
        // 0 <= floor < size as unsigned integers: false for negative, huge and NaN positions too
        inside = ux < (uint32_t)p.mov.w && uy < (uint32_t)p.mov.h;
        const uint32_t i = inside ? uy * (uint32_t)p.mov.w + ux : 0u;
        ax = pos.x - (tx - kMagic);
        ay = pos.y - (ty - kMagic);
        af = lam - (tl - kMagic);
        const uint32_t j = frow + (__float_as_uint(tl) - kBits);
#pragma unroll
        for (int c = 0; c < C; c++) {
            m[c] = __ldg(p.mov_quad + c * p.quad_plane + i);
            f[c] = __ldg(p.fix_pair + c * p.pair_plane + j);
        }
    }
    template <int COST>
    __device__ __forceinline__ void add(float &out, float2 &i12) const {
        const float2 s2 = make_float2(1.0f / 255.0f, 1.0f / 255.0f);
#pragma unroll
        for (int c = 0; c < C; c++) {
            const float2 tb = __ffma2_rn(make_float2(ax, ax), make_float2(m[c].z, m[c].w), make_float2(m[c].x, m[c].y));
            const float v = fmaf(ay, tb.y - tb.x, tb.x);
            const float2 w = __fmul2_rn(make_float2(inside ? v : 0.0f, fmaf(af, f[c].y, f[c].x)), s2);
            if constexpr (COST == CGS_COST_NCC_ALT) {
                out = fmaf(w.x, w.y, out);
            } else {
                const float d = w.x - w.y;
                out = fmaf(d, d, out);
            }
            i12 = __ffma2_rn(w, w, i12);
        }
    }
};

// calcNCCAlt and calcSQDAlt.  6,561 points on a 320 x 240 RGB pair take 1.73 ms (19 % of the L1's load
// instructions, 53 % of its wavefronts -- a quad load is four of them at best -- and 53 % of the issue
// slots; the rest is latency and the last points' tail).  Eight scalar taps a sample and channel, runs
// looked up for every sample and one CTA of 8 warps on an SM (84 KB of runs) took 7.95 ms.  Three CTAs fit
// here; two samples a lane are in flight, added in the lambda order.
template <int COST, int C>
__global__ void __launch_bounds__(kScanWarps * 32, 3) scan_sum_kernel(const __grid_constant__ SearchParams p) {
    constexpr bool kNCC = (COST == CGS_COST_NCC_ALT);
    constexpr int kStride = kMaxUnitSegs + 1;  // odd: the lanes' rows start in different banks
    __shared__ unsigned long long wbest[kScanWarps];
    __shared__ SumRow rows_all[kScanWarps][kScanRows];
    __shared__ uint2 segs_all[kScanWarps][kScanRows * kStride];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    SumRow *rows = rows_all[warp];
    uint2 *segs = segs_all[warp];
    const int fw = p.fix.w, fh = p.fix.h, mw = p.mov.w, mh = p.mov.h;
    const float fwf = (float)fw;
    // -0 the compiler cannot see: a product with it stays apart from the sum that follows
    const float nzero = __uint_as_float(0x80000000u | ((uint32_t)p.dims >> 8));
    const float2 nzero2 = make_float2(nzero, nzero);

    unsigned long long best = ~0ull;
    const uint32_t total_warps = gridDim.x * kScanWarps;
    for (uint32_t o = blockIdx.x * kScanWarps + warp; o < p.n; o += total_warps) {
        int32_t ax[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        const uint32_t gidx = ordinal_to_index(p, o, ax);
        float q[8];
        grid_values(p, ax, q);
        const float2 cs = p.trig[min(ax[0], kMaxTrig - 1)];
        const Homog H = h_centred(q, cs.x, cs.y, p.cx, p.cy);

        float out = 0.0f;                          // lane partial sums
        float2 i12 = make_float2(0.0f, 0.0f);
        double mov_area_d = 0.0;                   // sum n_r * mag_r
        uint32_t steps = 0;                        // lambda steps over all rows
        for (int rb = 0; rb < fh; rb += kScanRows) {
            const int nb = min(kScanRows, fh - rb);
            __syncwarp();
            if (lane < nb) {
                SumRow r;
                float le = fwf;
                r.ls = r.vx = r.vy = r.p0x = r.p0y = 0.0f;
                bool in = false;
                assign_values(H, mw, mh, fw, fh, rb + lane, r.ls, le, r.vx, r.vy, r.p0x, r.p0y, in);
                r.mag = __fsqrt_rn(xa(xm(r.vx, r.vx), xm(r.vy, r.vy)));
                r.nseg = 0;
                r.n = in ? unit_segments(r.ls, fminf(le, fwf), segs + lane * kStride, r.nseg) : 0u;
                rows[lane] = r;
            }
            __syncwarp();
            for (int rr = 0; rr < nb; rr++) {
                const SumRow r = rows[rr];
                if (r.n == 0) continue;
                steps += r.n;
                mov_area_d += (double)r.n * (double)r.mag;
                const uint32_t frow = (uint32_t)(rb + rr) * (uint32_t)fw;
                if (r.nseg > kMaxUnitSegs) {
                    float lam = r.ls;
                    if (lane < (int)r.n) seq_advance(lam, 1.0, (uint32_t)lane);
                    for (uint32_t k = lane; k < r.n; k += 32) {
                        SumSample<C> s;
                        s.load(p, r, nzero2, lam, frow);
                        s.template add<COST>(out, i12);
                        if (k + 32 < r.n) seq_advance(lam, 1.0, 32);
                    }
                    continue;
                }
                const uint2 *next = segs + rr * kStride, *last = next + r.nseg;
                uint2 cur = make_uint2(0u, 0u);
                uint32_t knext = 0u;  // index where the run after the current one begins
                float lam = 0.0f;     // lambda of sample k
                auto seek = [&](uint32_t k) {  // lam of sample k, from the one 32 before it within a run
                    lam += 32.0f;
                    if (k >= knext) {
                        do {
                            cur = *next++;
                            knext = next < last ? next->x : 0xffffffffu;
                        } while (k >= knext);
                        lam = __uint_as_float(cur.y) + (float)(k - cur.x);
                    }
                };
                uint32_t k = lane;
                for (; k - lane + 64 <= r.n; k += 64) {  // uniform: two full warps of samples
                    SumSample<C> s0, s1;
                    seek(k);
                    s0.load(p, r, nzero2, lam, frow);
                    seek(k + 32);
                    s1.load(p, r, nzero2, lam, frow);
                    s0.template add<COST>(out, i12);
                    s1.template add<COST>(out, i12);
                }
                for (; k < r.n; k += 32) {
                    SumSample<C> s;
                    seek(k);
                    s.load(p, r, nzero2, lam, frow);
                    s.template add<COST>(out, i12);
                }
            }
        }

        out = warp_sum(out);
        const float i1 = warp_sum(i12.x), i2 = warp_sum(i12.y);
        // gates (cudaErrorFunctions.cuh:296, 372): fix_area counts lambda steps exactly;
        // mov_area is a float running sum, decided from its double value unless that is
        // within the float sum's error bound of the threshold, then replayed exactly
        const float fix_area = (float)steps;
        const float den_m = xm((float)(p.mov.w * p.mov.h), q[2]);
        const bool gate_fix = (double)xd(fix_area, (float)(fw * fh)) > 0.35;
        bool gate_mov = false;
        if (lane == 0) {
            const double ratio = mov_area_d / (double)den_m;
            const double margin = ((double)steps + 4.0) * 5.9604644775390625e-8 * fabs(ratio) + 1e-12;
            if (fabs(ratio - 0.25) > margin) {
                gate_mov = ratio > 0.25;
            } else {
                // exact replay of the reference's sequential float sum
                float mov_area = 0.0f;
                for (int r = 0; r < fh; r++) {
                    float ls = 0.0f, le = fwf, vx = 0, vy = 0, p0x = 0, p0y = 0;
                    bool in = false;
                    assign_values(H, mw, mh, fw, fh, r, ls, le, vx, vy, p0x, p0y, in);
                    if (!in) continue;
                    bool st;
                    const uint32_t n = seq_count_below(ls, 1.0, fminf(le, fwf), st);
                    const float mag = __fsqrt_rn(xa(xm(vx, vx), xm(vy, vy)));
                    seq_advance(mov_area, (double)mag, n);
                }
                gate_mov = (double)xd(mov_area, den_m) > 0.25;
            }
            const float cost = gate_mov && gate_fix ? xd(kNCC ? -out : out, __fsqrt_rn(xm(i1, i2))) : 123123.0f;
            if (p.costs) p.costs[gidx] = cost;
            const unsigned long long kk = make_key(cost, gidx);
            best = kk < best ? kk : best;
        }
    }

    if (lane == 0) wbest[warp] = best;
    __syncthreads();
    if (threadIdx.x == 0) scan_finish(p, wbest);
}

// calcMIAlt.
template <int C>
__global__ void __launch_bounds__(kScanWarps * 32, 1) scan_kernel(const __grid_constant__ SearchParams p) {
    constexpr int NW = kScanWarps;
    constexpr int BN = 64;                 // calcMIAlt's bins
    constexpr int HS = BN + 1;             // padded row stride; row / column BN hold the marginals
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned long long *wbest = reinterpret_cast<unsigned long long *>(smem);
    RowInfo *rows_all = reinterpret_cast<RowInfo *>(smem + 8 * NW);
    Seg *segs_all = reinterpret_cast<Seg *>(rows_all + NW * kScanRows);
    uint32_t *hist_all = reinterpret_cast<uint32_t *>(segs_all + NW * kScanRows * kMaxSegs);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    RowInfo *rows = rows_all + warp * kScanRows;
    Seg *segs = segs_all + warp * kScanRows * kMaxSegs;
    uint32_t *hist = hist_all + (size_t)warp * HS * HS;
    const int fw = p.fix.w, fh = p.fix.h, mw = p.mov.w, mh = p.mov.h;
    const float fwf = (float)fw, fhf = (float)fh, mwf = p.mov_wf, mhf = p.mov_hf;
    const int nrows = p.n_rows;
    const double lam_inc = (double)(1.0f / (float)(fw - 1));

    unsigned long long best = ~0ull;
    const uint32_t total_warps = gridDim.x * NW;
    for (uint32_t o = blockIdx.x * NW + warp; o < p.n; o += total_warps) {
        int32_t ax[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        const uint32_t gidx = ordinal_to_index(p, o, ax);
        float q[8];
        grid_values(p, ax, q);
        const float2 cs = p.trig[min(ax[0], kMaxTrig - 1)];
        const Homog H = h_norm(q, cs.x, cs.y, mw, mh, fw, fh);

        uint32_t steps = 0;  // lambda steps over all rows (uniform)
        bool stalled = false;
        for (int i = lane; i < HS * HS; i += 32) hist[i] = 0u;
        __syncwarp();

        for (int rb = 0; rb < nrows; rb += kScanRows) {
            const int nb = min(kScanRows, nrows - rb);
            if (lane < nb) {
                RowInfo ri;
                ri.ls = 0.0f;
                ri.le = 1.0f;
                ri.vx = ri.vy = ri.p0x = ri.p0y = 0.0f;
                bool in = false;
                const float rv = p.row_table[rb + lane];
                assign_values_norm(H, rv, ri.ls, ri.le, ri.vx, ri.vy, ri.p0x, ri.p0y, in);
                ri.rowv = __double2float_rn(((double)rv + 0.5) * (double)(fh - 1));
                bool st = false, ovf = false;
                ri.nseg = 0;
                ri.n = in ? seq_segments(ri.ls, lam_inc, fminf(ri.le, 1.0f), segs + lane * kMaxSegs, kMaxSegs,
                                         ri.nseg, ovf, st)
                          : 0u;
                if (ovf) ri.nseg = -1;
                // a row has at most about W_f / step samples; anything else is a stalled
                // recurrence the reference would never leave
                const double max_n = (double)fw / fmin(lam_inc, 1.0) + 8.0;
                if ((double)ri.n > max_n) st = true;
                if (st) ri.n = 0u;
                rows[lane] = ri;
                stalled |= st;
            }
            __syncwarp();
            for (int rr = 0; rr < nb; rr++) {
                const RowInfo ri = rows[rr];
                if (ri.n == 0) continue;
                steps += ri.n;
                const Seg *rs = segs + rr * kMaxSegs;
                int cur = 0;
                float lam = ri.ls;
                bool ok = true;
                if (ri.nseg < 0 && lane < (int)ri.n) ok = seq_advance(lam, lam_inc, (uint32_t)lane);
                for (uint32_t k = lane; k < ri.n; k += 32) {
                    if (ri.nseg >= 0) lam = seq_value(rs, ri.nseg, cur, k);
                    const float nx0 = xa(xm(lam, ri.vx), ri.p0x);
                    const float ny0 = xa(xm(lam, ri.vy), ri.p0y);
#pragma unroll
                    for (int c = 0; c < C; c++) {
                        const float *mpl = p.mov.data + c * p.mov.plane;
                        const float *fpl = p.fix.data + c * p.fix.plane;
                        const float nx = __double2float_rn(((double)nx0 + 0.5) * (double)mw);
                        const float ny = __double2float_rn(((double)ny0 + 0.5) * (double)mh);
                        const float lamIdx = xm(lam, (float)(fw - 1));
                        const float vf = value_exact(fpl, p.fix.pitch, fwf, fhf, ri.rowv, lamIdx);
                        const float vm = value_exact(mpl, p.mov.pitch, mwf, mhf, ny, nx);
                        int bf = (int)floorf(xm(64.0f, xd(vf, 256.0f)));
                        int bm = (int)floorf(xm(64.0f, xd(vm, 256.0f)));
                        bf = min(max(bf, 0), BN - 1);
                        bm = min(max(bm, 0), BN - 1);
                        atomicAdd(&hist[bf * HS + bm], 1u);
                    }
                    if (ri.nseg < 0 && k + 32 < ri.n) ok &= seq_advance(lam, lam_inc, 32);
                }
                stalled |= !ok;
            }
            __syncwarp();
        }

        // ---- cost of this grid point
        // marginals: fixed (rows) into column BN, moving (columns) into row BN
        for (int i = lane; i < BN; i += 32) {
            uint32_t rs = 0, csum = 0;
            for (int j = 0; j < BN; j++) {
                rs += hist[i * HS + j];
                csum += hist[j * HS + i];
            }
            hist[i * HS + BN] = rs;
            hist[BN * HS + i] = csum;
        }
        __syncwarp();
        uint32_t cnt = 0;
        for (int i = lane; i < BN; i += 32) cnt += hist[i * HS + BN];
        cnt = (uint32_t)warp_sum_i((int)cnt);
        // the reference's float formula: P = n_xy / count, sum P (log2 P - (log2 Px + log2 Py))
        const float countf = (float)cnt;
        float s = 0.0f;
        for (int b = lane; b < BN * BN; b += 32) {
            const int i = b / BN, j = b - i * BN;
            const uint32_t v = hist[i * HS + j];
            if (v) {
                const float P = (float)v / countf;
                const float Px = (float)hist[i * HS + BN] / countf;
                const float Py = (float)hist[BN * HS + j] / countf;
                s += P * (log2f(P) - (log2f(Px) + log2f(Py)));
            }
        }
        s = warp_sum(s);
        // fix_area: one 1/(W_f H_f) per lambda step, accumulated as the reference does
        float fix_area = 0.0f;
        seq_advance(fix_area, 1.0 / (double)((int64_t)fw * fh), steps);
        const float cost = (-1.0f * s) * fix_area;
        stalled = __any_sync(0xffffffffu, stalled);
        if (lane == 0) {
            if (stalled) atomicOr(p.status, (unsigned)CGS_ERROR_UNSUPPORTED);
            if (p.costs) p.costs[gidx] = cost;
            const unsigned long long kk = make_key(cost, gidx);
            best = kk < best ? kk : best;
        }
        __syncwarp();
    }

    if (lane == 0) wbest[warp] = best;
    __syncthreads();
    if (threadIdx.x == 0) scan_finish(p, wbest);
}

}  // namespace cgs
