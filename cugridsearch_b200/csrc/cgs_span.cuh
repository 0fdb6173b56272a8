// cgs_span.cuh -- the span kernel: zero-mean NCC over fast samples, with the in/out decisions
// taken per image row instead of per sample, the moving image's taps read from shared memory,
// and the fixed image's sums read from row prefix sums.  Its staging step is span_prep_kernel
// (end of this file), after the shared staging kernel has written the span form of the quads.
//
// Decisions per row.  For one grid point the map of a fixed row y is a projective line in the
// moving image; the samples that lie inside the moving image form one interval of x.  Solving
// the four half-plane conditions of "clearly inside" (a margin of 1.5 guard bands inside the
// image's edges, the guard being map_guard's bound between the fast and the reference's
// coordinates) and of "possibly inside" (1.5 guard bands outside) gives two integer spans per
// (row, point): every pixel of the inner span is inside for the reference too and takes the
// fast path with no test; pixels of the outer span outside the inner one (a band about a
// thousandth of a pixel wide around the overlap's edge, almost never a whole pixel) take the
// reference's exact operation sequence, evaluated once per band of rows by the lane that
// computed the span; every other pixel is outside and costs nothing.  The spans are computed
// in FP32; their rounding error is below a quarter of the guard band (the constraint terms are
// those the guard's own bound is built from), which the 1.5 factor covers.
//
// Fixed-image sums.  sum f and sum f^2 over a point's overlap are the inner spans' sums, taken
// from FP64 prefix sums of each fixed row (span_prep_kernel; where a pixel before the span swamps
// them, from the pixels: prefix_holds), plus the band pixels found inside; only the three sums that
// involve the moving image are accumulated per sample.
//
// Tiles and windows.  The fixed image is walked in tiles of TW = 32 TX columns by TH rows.  For
// every 32-column block of a tile the CTA's grid points map the block into a small region of
// the moving image (the union of the block's quadrilateral images, points of one task being
// neighbours in the locality order); the regions of a tile's blocks are copied from the staged
// tap quads into the window stage by bulk copies, one per region row, and the sweep reads its
// 16-byte quads from there.  A block whose region does not fit the stage reads global memory
// instead (same values).  Blocks rather than whole tiles bound the regions of rotated maps.
//
// One stage, filled by every warp.  The stage takes all the shared memory that is left (about
// 12 K quads), which holds the eight windows of a 256 x 16 tile at +-20 degrees (8-11 K quads);
// two stages of half the size sent a third of the blocks to global memory.  The next tile's
// copies start at the barrier that ends a tile and run during the next band's span pass; a tile's
// wait is then 0.5-2 K cycles of about 65 K.  Measured on the 256 x 256, 6^8 search: two stages
// filled by one warp 133.3 ms, one stage filled by one warp 128.6 ms, by all warps 116.1 ms (105.8 ms with
// the cheaper task setup and span pass that came after).
//
// Sweep.  Lane l takes the tile's columns x0 + l + 32 k; each warp evaluates its G grid points
// at every pixel, two points per packed FP32x2 instruction.  Blocks inside every point's inner
// span run without any per-sample test; other blocks mask samples by the inner spans.  A
// sample's quad index comes from the floor bits of its coordinates in one FP32x2 multiply-add
// (x + pitch y, exact below 2^22), its address from one shift-add.
//
// Sums.  Per lane, per band of TH rows: three FP32 sums per point of the shifted values
// f' = f - s_f, m' = m - s_m (the images' means; sum m', sum m'^2, sum f'm'), reduced across the
// warp at the end of each band of tiles and accumulated in FP64 with the spans' fixed-image
// sums and the band pixels' sums; the cost is formed in FP64 (zncc_cost).  Which samples a lane
// sums, and in which order, depends only on the image and the tile shape, never on the points
// per warp or the warps per CTA: costs are bit-identical across those tunings.  The overlap
// count is the sum of the inner span lengths plus the band pixels found inside.
#pragma once
#include <cstddef>
#include <type_traits>

#include "cgs_kernels.cuh"

namespace cgs {

// Moving images with (W + 8) H >= 2^22 are outside the span path: the quad index x + pitch y
// (pitch at most W + 7) is formed exactly in FP32 below that.
constexpr int64_t kSpanMaxQuads = (int64_t)1 << 22;
// kStatusSpanBounds (cgs_internal.h): status bit the self-checking build (CHECK = true) sets in
// the result when a fast sample's quad address fell outside its block's window or the quad
// plane (the sample is then skipped).

// Everything the span path keeps of one grid point (shared memory, one per point of the task).
struct SpanSlot {
    float A, B, PQ, C1, C2, RS, D1, D2, TU;  // fast map: w = A x + (B y + PQ), X = .., Y = ..
    float P, Q, R, S, T, U;                  // exact-path terms (with A, B, C1, C2, D1, D2)
    float gx, gy;                            // guard band (map_guard)
    int32_t ok;                              // 1: fast path valid (guard holds, point in the grid)
    int32_t valid;                           // 1: ordinal inside the grid
    uint32_t index;                          // grid index of the point
};

// Row-term coefficients of a pair of points, packed for FP32x2: {B, PQ, C2, RS, D2, TU} of
// point 2h and 2h + 1 interleaved.
struct PairRow {
    float2 B, PQ, C2, RS, D2, TU;
};

// The moving-image window of one 32-column block of a tile: quads [y0, y0 + h) x [x0, x0 + w)
// with row pitch `pitch` quads, `off` quads into the stage's window area; h == 0: no point
// samples the block on the fast path; w < 0: the window does not fit the stage and the sweep
// reads global memory.  For the sweep: rel = 16 (off - x0 - pitch y0 - kMagicBits) (mod 2^32),
// so that quad (ix, iy) lies at stage window + rel + 16 bits(tx - nfy pitch); pitchf = -pitch.
struct BlockWin {
    int16_t x0, y0, w, h;
    int32_t pitch, off;
    uint32_t rel;
    float pitchf;
};
static_assert(sizeof(BlockWin) == 24 && offsetof(BlockWin, rel) == 16, "the sweep reads {rel, pitchf} as 8 bytes");

// Inner span of one (point, row): [xa, xa + len).
struct InnerSpan {
    int32_t xa, len;
};

// One row of a warp's points: [ia, ib] lies in every point's inner span (empty if ia > ib),
// [ua, ub] is the hull of their inner spans (empty if ua > ub).
struct RowRun {
    int32_t ia, ib, ua, ub;
};

__host__ __device__ constexpr size_t span_head_bytes(int NW) { return 256 + 8 * (size_t)NW; }

// Shared-memory plan of the span kernel for NW warps of G points, TH-row bands, tiles of TX
// blocks, `tiles` tiles and a stage of `cap` quads.
__host__ __device__ constexpr size_t span_smem_bytes(int G, int NW, int TH, int TX, int tiles, int cap) {
    return span_head_bytes(NW) + (size_t)NW * G * sizeof(SpanSlot) + (size_t)NW * (G / 2) * sizeof(PairRow) +
           (size_t)tiles * TX * sizeof(BlockWin) + (size_t)NW * G * TH * sizeof(InnerSpan) +
           (size_t)NW * TH * sizeof(RowRun) + (size_t)NW * G * (10 * sizeof(double) + sizeof(int)) +
           (size_t)cap * 16 + 144;
}

struct SpanSmem {
    uint64_t *bar;     // the window stage's barrier
    unsigned long long *wbest;
    int *abort_flag;
    int *bounds_flag;  // self-checking build: a sample's quad address fell outside its window
    SpanSlot *slots;   // [NW * G]
    PairRow *prow;     // [NW * G / 2]
    BlockWin *wins;    // [tiles][TX]
    InnerSpan *spans;  // [NW][G][TH]
    RowRun *runs;      // [NW][TH]
    double *dtot;      // [NW][G * 5] FP64 task totals {sum f, sum m', sum f^2, sum m'^2, sum f'm'}
    double *dband;     // [NW][G * 5] the same sums of the current band
    int *cnt;          // [NW][G] overlap counts of the warps' points
    float4 *win;       // [cap] the window stage
    int cap;
    float2 *rowtab;    // exact span kernel: [NW][TH][G / 2][3] products of the rows
    uint32_t *hist;    // exact span kernel, MI: [NW * G][(B + 1)^2]
};

// `exact`: the exact span kernel's row products, and histograms of mi_bins bins (0: none), before the stage.
template <int G, int NW>
__device__ __forceinline__ SpanSmem carve_span(unsigned char *smem, int TH, int TX, int tiles, int cap,
                                               bool exact = false, int mi_bins = 0) {
    SpanSmem s;
    s.bar = reinterpret_cast<uint64_t *>(smem);
    s.wbest = reinterpret_cast<unsigned long long *>(smem + 64);
    s.abort_flag = reinterpret_cast<int *>(smem + 64 + 8 * NW);
    s.bounds_flag = s.abort_flag + 1;
    unsigned char *q = smem + span_head_bytes(NW);
    s.slots = reinterpret_cast<SpanSlot *>(q);
    q += (size_t)NW * G * sizeof(SpanSlot);
    s.prow = reinterpret_cast<PairRow *>(q);
    q += (size_t)NW * (G / 2) * sizeof(PairRow);
    s.wins = reinterpret_cast<BlockWin *>(q);
    q += (size_t)tiles * TX * sizeof(BlockWin);
    s.spans = reinterpret_cast<InnerSpan *>(q);
    q += (size_t)NW * G * TH * sizeof(InnerSpan);
    s.runs = reinterpret_cast<RowRun *>(q);
    q += (size_t)NW * TH * sizeof(RowRun);
    s.dtot = reinterpret_cast<double *>(q);
    q += (size_t)NW * G * 5 * sizeof(double);
    s.dband = reinterpret_cast<double *>(q);
    q += (size_t)NW * G * 5 * sizeof(double);
    s.cnt = reinterpret_cast<int *>(q);
    q += (size_t)NW * G * sizeof(int);
    s.rowtab = reinterpret_cast<float2 *>(smem + (((size_t)(q - smem) + 15) & ~(size_t)15));
    s.hist = nullptr;
    if (exact) {
        q = reinterpret_cast<unsigned char *>(s.rowtab) + (((size_t)NW * TH * (G / 2) * 24 + 15) & ~(size_t)15);
        s.hist = reinterpret_cast<uint32_t *>(q);
        if (mi_bins > 0) q += ((size_t)NW * G * (mi_bins + 1) * (mi_bins + 1) * 4 + 15) & ~(size_t)15;
    }
    // aligned by offset from the shared base (an integer round trip of the pointer would lose
    // its shared-memory provenance and turn every window read into a generic load)
    const size_t off = ((size_t)(q - smem) + 127) & ~(size_t)127;
    s.win = reinterpret_cast<float4 *>(smem + off);
    s.cap = cap;
    return s;
}

// Spans of one row of one point: the inner span [xa, xa + len) and the outer span [pa, pa + plen),
// which holds it.
struct RowSpans {
    int xa, len, pa, plen;
};
constexpr int kFewBand = 8;  // band pixels of a row that its lane samples by itself (exact costs, MI)

// The spans of row y (see the head of this file).  Each edge of the moving image gives a condition
// s f(x) > 0 with f(x) = a x + b linear and s the sign of w; x = q solves f = 0.  f is the distance
// to the edge in pixels times w, so with h = 1.5 g max|w| / |a| (max over the row) every x beyond
// q + h lies at least 1.5 guard bands inside that edge and every x beyond q - h at least as far
// outside it: one reciprocal gives both spans.  An edge that the row follows (a changes f by less
// than a thousandth of the margin over the whole row) is decided by b alone.  Branch-free: the
// reciprocals of the four edges overlap (IEEE divisions, one per edge and span, took 40 % of the
// span pass).
__device__ __forceinline__ RowSpans row_spans(const SpanSlot &k, float yf, int fw, float mw, float mh) {
    const float bw = fmaf(k.B, yf, k.PQ), bX = fmaf(k.C2, yf, k.RS), bY = fmaf(k.D2, yf, k.TU);
    const float fwf = (float)fw, we = fmaf(k.A, fwf - 1.0f, bw);
    const float s = bw > 0.0f ? 1.0f : -1.0f;  // the guard holds: w keeps its sign over the image
    const float wmax = fmaxf(fabsf(bw), fabsf(we));
    float ilo = -1.0f, ihi = fwf, olo = -1.0f, ohi = fwf;  // open intervals, clamped to the row
    bool inone = false, onone = false;
    auto edge = [&](float a, float b, float m) {  // m: the margin times max|w|
        a *= s;
        b *= s;
        const bool flat = fabsf(a) * fwf < 1e-3f * m;
        const float r = rcp_approx(a);
        const float q0 = -b * r;
        const float q = fmaf(fmaf(-q0, a, -b), r, q0), h = m * fabsf(r);
        const bool up = !flat && a > 0.0f, down = !flat && a < 0.0f;
        ilo = up ? fmaxf(ilo, q + h) : ilo;
        olo = up ? fmaxf(olo, q - h) : olo;
        ihi = down ? fminf(ihi, q - h) : ihi;
        ohi = down ? fminf(ohi, q + h) : ohi;
        inone = inone || (flat && !(b > 1.01f * m));
        onone = onone || (flat && !(b > -1.01f * m));
    };
    const float gx = 1.5f * k.gx * wmax, gy = 1.5f * k.gy * wmax;
    edge(k.C1, bX, gx);                                    // X > 0
    edge(fmaf(mw, k.A, -k.C1), fmaf(mw, bw, -bX), gx);     // W w - X > 0
    edge(k.D1, bY, gy);                                    // Y > 0
    edge(fmaf(mh, k.A, -k.D1), fmaf(mh, bw, -bY), gy);     // H w - Y > 0
    ilo = fmaxf(ilo, -1.0f);
    olo = fmaxf(olo, -1.0f);
    const int a0 = max(0, (int)floorf(fminf(ilo, fwf)) + 1), b0 = min(fw - 1, (int)ceilf(fmaxf(ihi, -1.0f)) - 1);
    const int a1 = max(0, (int)floorf(fminf(olo, fwf)) + 1), b1 = min(fw - 1, (int)ceilf(fmaxf(ohi, -1.0f)) - 1);
    RowSpans r;
    r.xa = a0;
    r.len = (inone || b0 < a0) ? 0 : b0 - a0 + 1;
    r.pa = a1;
    r.plen = (onone || b1 < a1) ? 0 : b1 - a1 + 1;
    return r;
}

// Prefix sums stand for the sums of an inner span only where the span's sum of squares d is not lost in the
// rounding of the prefix `to` that it was taken from: a pixel before the span that is not finite or far
// larger poisons the difference, and a span of zeros must sum to 0 exactly.  The sum of f, at most
// sqrt(W) times the root of that of squares, is then safe too.  Above 2^-16 of the prefix the
// error, at most (5 + W / 32) 2^-53 of it, is below 2^-27 of the sum; below that the pixels are added
// (row_sums).  Images without such pixels have next to no rows there.
__device__ __forceinline__ bool prefix_holds(double d, double to) { return d > 0x1p-16 * to || to == 0.0; }

// {sum f, sum f^2} over the channels of pixels [xa, xa + len) of fixed row y, by the whole warp.
template <int C>
__device__ __noinline__ double2 row_sums(const Plane &fix, int y, int xa, int len) {
    double s1 = 0.0, s2 = 0.0;
    const float *row = fix.data + (int64_t)y * fix.pitch + xa;
    for (int i = threadIdx.x & 31; i < len; i += 32)
#pragma unroll
        for (int ch = 0; ch < C; ch++) {
            const double f = (double)__ldg(row + ch * fix.plane + i);
            s1 += f;
            s2 += f * f;
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    return make_double2(s1, s2);
}

// The corners of block [x0, x1] x [y0, y1] under a point's map: min/max of the mapped coordinates.
__device__ __forceinline__ void block_extent(const SpanSlot &k, float x0, float x1, float y0, float y1, float4 &e) {
    auto one = [&](float x, float y) {
        const float w = fmaf(k.A, x, fmaf(k.B, y, k.PQ));
        const float X = fmaf(k.C1, x, fmaf(k.C2, y, k.RS));
        const float Y = fmaf(k.D1, x, fmaf(k.D2, y, k.TU));
        const float rw = rcp_approx(w), mx = X * rw, my = Y * rw;  // the 0.25 px margin covers their error
        e.x = fminf(e.x, mx);
        e.y = fminf(e.y, my);
        e.z = fmaxf(e.z, mx);
        e.w = fmaxf(e.w, my);
    };
    one(x0, y0);
    one(x1, y0);
    one(x0, y1);
    one(x1, y1);
}

// One count into a shared-memory histogram.  No compiler memory clobber: the counts are read only
// after a __syncwarp or __syncthreads, and the loads of the next samples may move ahead of it.
__device__ __forceinline__ void red_shared_add1(uint32_t addr) {
    asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(addr));
}

// The reference's bin of value v: min(max(floor(v B / 256), 0), B - 1).
__device__ __forceinline__ int mi_bin(float v, float sB, int B) { return min(max((int)floorf(v * sB), 0), B - 1); }

// Thread 0: announce the bytes of tile t's copies on the stage's barrier (its one arrival).  It
// comes before the CTA barrier after which every warp issues its part (issue_window).
template <int C, int TX>
__device__ __forceinline__ void expect_window(const SearchParams &p, const SpanSmem &ss, int t) {
    constexpr int TW = 32 * TX;
    const int x0 = (t % p.tiles_x) * TW, y0 = (t / p.tiles_x) * p.tile_h;
    const BlockWin *bw = ss.wins + t * TX;
    uint32_t bytes = (uint32_t)min(p.tile_h, p.fix.h - y0) * (uint32_t)((min(TW, p.fix.w - x0) * 4 + 15) & ~15);
#pragma unroll
    for (int c = 0; c < TX; c++)
        if (bw[c].h > 0 && bw[c].w > 0) bytes += (uint32_t)bw[c].w * (uint32_t)bw[c].h * 16u;
    bytes *= C;
    mbar_arrive_expect_tx(ss.bar, bytes);
}

// Issue (every warp its part) the copies of tile t into the stage, completing on its
// barrier: the tile's rows of the fixed plane(s) fsrc, of p.fix's pitch (TH x TW floats at the stage's start; columns
// past the image's right edge are not copied) and the windows of its blocks (quads, after the
// fixed tile).  A tile has about 220 row copies and a warp issues one in about 60 cycles, so one
// warp would hold the others back for 14 K cycles per tile; shared by the CTA's warps it is 1 K.
template <int C, int NW, int TX>
__device__ __forceinline__ void issue_window(const SearchParams &p, const SpanSmem &ss, const float *fsrc, int t) {
    constexpr int TW = 32 * TX;
    constexpr int WB = NW / TX;  // warps per block window
    static_assert(NW % TX == 0, "whole warps per block window");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int TH = p.tile_h;
    const int x0 = (t % p.tiles_x) * TW, y0 = (t / p.tiles_x) * TH;
    uint64_t *bar = ss.bar;
    fence_proxy_async_smem();  // the stage's previous reads before the async refill
    if (lane == 31) {
        const int rows = min(TH, p.fix.h - y0);
        const uint32_t row_bytes = (uint32_t)((min(TW, p.fix.w - x0) * 4 + 15) & ~15);  // within the row pitch
        float *fdst = reinterpret_cast<float *>(ss.win);
        for (int j = warp; j < rows; j += NW)
#pragma unroll
            for (int ch = 0; ch < C; ch++)
                bulk_g2s(fdst + (ch * TH + j) * TW, fsrc + ch * p.fix.plane + (int64_t)(y0 + j) * p.fix.pitch + x0,
                         row_bytes, bar);
    }
    const BlockWin b = ss.wins[t * TX + warp / WB];
    if (b.h > 0 && b.w > 0) {
        float4 *wdst = ss.win + C * TH * TW / 4 + b.off;
        const float4 *src = p.mov_quad + (int64_t)b.y0 * p.quad_pitch + b.x0;
        for (int j = lane * WB + warp % WB; j < b.h; j += 32 * WB)
#pragma unroll
            for (int ch = 0; ch < C; ch++)
                bulk_g2s(wdst + (size_t)(ch * b.h + j) * b.pitch, src + ch * p.quad_plane + (int64_t)j * p.quad_pitch,
                         (uint32_t)b.w * 16u, bar);
    }
}

// Correctly rounded quotients without a branch: x = X / w and y = Y / w of a pair of points from w,
// -X and -Y (the caller forms the negatives by negating coefficients, which is exact).  The reciprocal
// r of w is the approximate one and a Newton step; the quotient q0 = X r is corrected by its exact
// residual, q = q0 + (X - w q0) r (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990).  r and q are the correctly rounded values, provided
// that no step leaves the normal range (quot_range): one run over every pair of 24-bit mantissas (2^46
// quotients) found none that differs from IEEE division; tests/native/span_check.cu repeats 3.9e9 of them.  Eight packed operations and two reciprocals replace four
// divisions of about ten instructions and a branch each.
__device__ __forceinline__ void exact_quot2(float2 w, float2 nX, float2 nY, float2 &x, float2 &y) {
    const float2 nr0 = make_float2(rcp_approx(-w.x), rcp_approx(-w.y));
    const float2 e = __ffma2_rn(w, nr0, make_float2(1.0f, 1.0f));
    const float2 nr = __ffma2_rn(e, nr0, nr0);
    const float2 x0 = __fmul2_rn(nX, nr), y0 = __fmul2_rn(nY, nr);
    x = __ffma2_rn(__ffma2_rn(w, x0, nX), nr, x0);
    y = __ffma2_rn(__ffma2_rn(w, y0, nY), nr, y0);
}

// Whether exact_quot2 applies to every pixel of a fw x fh image: |w| in [2^-40, 2^40] at the corners
// (w is linear and the guard keeps its sign), numerators below 2^60, and every numerator coefficient
// zero or at least 2^-70, so that a numerator, a sum of multiples of 2^-93, is zero or at least that.
__device__ __forceinline__ bool quot_range(const MapCoef &k, int fw, int fh) {
    const float x1 = (float)(fw - 1), y1 = (float)(fh - 1), pq = k.P - k.Q;
    const float w0 = fabsf(pq), w1 = fabsf(k.A * x1 + pq), w2 = fabsf(k.B * y1 + pq), w3 = fabsf(k.A * x1 + k.B * y1 + pq);
    bool ok = fminf(fminf(w0, w1), fminf(w2, w3)) >= 0x1p-40f && fmaxf(fmaxf(w0, w1), fmaxf(w2, w3)) <= 0x1p40f;
    const float c[8] = {k.C1, k.C2, k.R, k.S, k.D1, k.D2, k.T, k.U};
#pragma unroll
    for (int i = 0; i < 8; i++) ok = ok && (c[i] == 0.0f || (fabsf(c[i]) >= 0x1p-70f && fabsf(c[i]) <= 0x1p40f));
    return ok;
}

// The G grid points from ordinal ord0: lane g decodes point g and writes its slot (the decode, the
// homography and the FP64 guard of a point are a chain of about 5 K cycles: four at once).  `ok`: the
// guard holds and, for exact samples (EXACT), the point's quotients are in the range of exact_quot2.
template <int COST, int G, bool EXACT = false>
__device__ __forceinline__ void span_points(const SearchParams &p, uint32_t ord0, SpanSlot *slots) {
    const int lane = threadIdx.x & 31;
    if (lane >= G) return;
    const uint32_t o = ord0 + lane;
    const bool gvalid = o < p.n;
    int32_t ax[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const uint32_t gidx = gvalid ? ordinal_to_index(p, o, ax) : 0u;
    float q[8];
    grid_values(p, ax, q);
    const float2 cs = p.trig[min(ax[0], kMaxTrig - 1)];
    const MapCoef kc = make_coef<COST>(q, cs, p);
    FastMap fm;
    RowTerms rt;
    float gx, gy;
    const bool guard = map_guard(kc, p, fm, rt, gx, gy);
    const bool ok = gvalid && guard && (EXACT ? quot_range(kc, p.fix.w, p.fix.h) : fm.li_x > 0.0f);
    slots[lane] = SpanSlot{kc.A, rt.B, rt.PQ, kc.C1, rt.C2, rt.RS, kc.D1, rt.D2, rt.TU, kc.P, kc.Q, kc.R,
                           kc.S, kc.T, kc.U, gx, gy, ok ? 1 : 0, gvalid ? 1 : 0, gidx};
}

// The windows of every block of tiles t0 .. t1 - 1, into ss.wins: warp w takes blocks w, w + NW, .. with the
// task's points over its lanes, then one thread per tile lays its blocks out in the stage (C planes of
// quads each, pitch x h apart).
template <int C, int G, int NW, int TX>
__device__ __forceinline__ void span_windows(const SearchParams &p, const SpanSmem &ss, int t0, int t1) {
    constexpr int TW = 32 * TX;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int fw = p.fix.w, fh = p.fix.h, TH = p.tile_h, tiles_x = p.tiles_x;
    const float mov_wf = p.mov_wf, mov_hf = p.mov_hf;
    constexpr int P = NW * G;
    const float inf = __int_as_float(0x7f800000);
    for (int i = t0 * TX + warp; i < t1 * TX; i += NW) {
        const int t = i / TX, c = i - t * TX;
        const int xc = (t % tiles_x) * TW + 32 * c, y0 = (t / tiles_x) * TH;
        float4 e = make_float4(inf, inf, -inf, -inf);
        if (xc < fw) {
            const float fx0 = (float)xc, fx1 = (float)(min(xc + 32, fw) - 1);
            const float fy0 = (float)y0, fy1 = (float)(min(y0 + TH, fh) - 1);
            for (int k = lane; k < P; k += 32)
                if (ss.slots[k].ok) block_extent(ss.slots[k], fx0, fx1, fy0, fy1, e);
            e.x = warp_fmin(e.x);
            e.y = warp_fmin(e.y);
            e.z = warp_fmax(e.z);
            e.w = warp_fmax(e.w);
        }
        if (lane == 0) {  // the block's extent, in its window's place
            float2 *d = reinterpret_cast<float2 *>(&ss.wins[i]);
            d[0] = make_float2(e.x, e.y);
            d[1] = make_float2(e.z, e.w);
        }
    }
    __syncthreads();
    const int wcap = ss.cap - C * TH * TW / 4;  // quads of a stage after the fixed rows
    for (int t = t0 + threadIdx.x; t < t1; t += NW * 32) {
        int used = 0;
#pragma unroll 1
        for (int c = 0; c < TX; c++) {
            BlockWin bw{0, 0, 0, 0, 0, 0, 0u, 0.0f};
            // cells a fast sample can use: floor of its coordinate (within the guard, < 1/8 px,
            // of the real map, whose block image lies in the corners' hull), clipped to the image
            const float2 *d = reinterpret_cast<const float2 *>(&ss.wins[t * TX + c]);
            const float2 e0 = d[0], e1 = d[1];
            const float lx = fmaxf(e0.x - 0.25f, -1.0f), ly = fmaxf(e0.y - 0.25f, -1.0f);
            const float hx = fminf(e1.x + 0.25f, mov_wf), hy = fminf(e1.y + 0.25f, mov_hf);
            if (lx <= hx && ly <= hy) {
                const int cx0 = max(0, (int)floorf(lx)), cy0 = max(0, (int)floorf(ly));
                const int cx1 = min(p.mov.w - 1, (int)floorf(hx)), cy1 = min(p.mov.h - 1, (int)floorf(hy));
                if (cx0 <= cx1 && cy0 <= cy1) {
                    const int w = cx1 - cx0 + 1, h = cy1 - cy0 + 1;
                    const int pitch = w + ((p.win_pitch_mod - w) & 7);  // = win_pitch_mod (mod 8)
                    bw.x0 = (int16_t)cx0;
                    bw.y0 = (int16_t)cy0;
                    bw.h = (int16_t)h;
                    bw.pitch = pitch;
                    if ((int64_t)C * pitch * h <= wcap - used) {
                        bw.w = (int16_t)w;
                        bw.off = used;
                        bw.rel = 16u * ((uint32_t)used - (uint32_t)cx0 - (uint32_t)pitch * (uint32_t)cy0 -
                                        (uint32_t)kMagicBits);
                        bw.pitchf = -(float)pitch;
                        used += C * pitch * h;
                    } else {
                        bw.w = -1;
                    }
                }
            }
            ss.wins[t * TX + c] = bw;
        }
    }
}

// Split tasks.  With fewer tasks than a few per SM the last wave leaves SMs idle (324 tasks on 148 SMs
// take three waves for the work of 2.2), so the host splits every task's bands of rows into `splits`
// parts, one per CTA at a time (span_splits).  The totals of each band go to global memory, and the CTA
// that completes a task's parts adds them in band order: the sums, and their order, are those of an
// unsplit task.

constexpr unsigned kPartLost = 1u << 16;  // in a task's count of done parts: one more was not run

// The band's sums of a warp's points (my_band, cleared) into the task totals, or to global memory.
template <int G, int NW>
__device__ __forceinline__ void fold_band(const SearchParams &p, uint32_t task, int band, double *my_dtot, double *my_band) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncwarp();
    for (int i = lane; i < G * 5; i += 32) {
        const double v = my_band[i];
        my_band[i] = 0.0;
        if (p.splits > 1) p.split_tot[(((size_t)task * p.tiles_y + band) * NW + warp) * (G * 5) + i] = v;
        else my_dtot[i] += v;
    }
    __syncwarp();
}

// After a part's bands: whether this CTA completed the task, whose totals and counts it then holds.  The
// self-checking build's finding is reported for every part, before the part counts as done (a CTA
// barrier precedes the call).
template <int G, int NW, bool CHECK>
__device__ __forceinline__ bool join_parts(const SearchParams &p, uint32_t task, int part, const SpanSmem &ss, double *my_dtot,
                                           int *my_cnt) {
    if (CHECK && threadIdx.x == 0 && *ss.bounds_flag) atomicOr(p.status, kStatusSpanBounds);
    if (p.splits <= 1) return true;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int *cnt = p.split_cnt + (size_t)task * p.splits * (NW * G) + warp * G;
    if (lane < G) cnt[part * (NW * G) + lane] = my_cnt[lane];
    __threadfence();
    __syncthreads();
    volatile int &s_last = *(ss.bounds_flag + 2);
    if (threadIdx.x == 0) {
        const unsigned done = atomicAdd(p.split_done + task, 1u) + 1u;
        s_last = (done & (kPartLost - 1u)) == (unsigned)p.splits;
        if (s_last && done >= kPartLost) {  // totals are missing: the task has no costs
            retire_tasks(p, ~0ull, 1u, true);
            s_last = 0;
        }
    }
    __syncthreads();
    if (!s_last) return false;
    __threadfence();
    for (int i = lane; i < G * 5; i += 32) {
        const double *t = p.split_tot + ((size_t)task * p.tiles_y * NW + warp) * (G * 5) + i;
        double d = 0.0;
        for (int b = 0; b < p.tiles_y; b++) d += __ldcg(t + (size_t)b * (NW * G * 5));
        my_dtot[i] = d;
    }
    if (lane < G) {
        int n = 0;
        for (int k = 0; k < p.splits; k++) n += __ldcg(cnt + k * (NW * G) + lane);
        my_cnt[lane] = n;
    }
    __syncwarp();
    return true;
}

// Thread 0 of a CTA that stops: the parts it will not run count as done and lost (join_parts: nobody
// adds their totals), and a task whose parts are all done is retired with the timeout status.
__device__ __forceinline__ void retire_parts(const SearchParams &p, uint32_t unit, uint32_t step, uint32_t units) {
    for (uint32_t u = unit; u < units; u += step) {
        if (p.splits <= 1) {
            retire_tasks(p, ~0ull, 1u, true);
            continue;
        }
        atomicOr(p.status, (unsigned)CGS_ERROR_DEVICE_TIMEOUT);
        __threadfence();
        const unsigned done = atomicAdd(p.split_done + u / p.splits, kPartLost + 1u) + 1u;
        if ((done & (kPartLost - 1u)) == (unsigned)p.splits) retire_tasks(p, ~0ull, 1u, true);
    }
}

// One task, or part of a task, of the span path (ZNCC, one channel, quads staged): the G grid points of
// each warp over the part's tiles of the fixed image.  `wit` counts this CTA's tiles (the
// barrier's phases).  Returns false if a bounded wait gave up.
template <int G, int NW, int TX, bool CHECK>
__device__ __forceinline__ bool run_span_task(const SearchParams &p, uint32_t unit, const SpanSmem &ss,
                                              uint32_t &wit) {
    static_assert(G % 2 == 0, "the span path pairs grid points");
    constexpr int GP = G / 2;
    constexpr int TW = 32 * TX;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int fw = p.fix.w, fh = p.fix.h;
    const int TH = p.tile_h;
    const int tiles_x = p.tiles_x;
    const uint32_t task = unit / (uint32_t)p.splits;
    const int part = (int)(unit - task * (uint32_t)p.splits);
    const int t0 = part * p.tiles_y / p.splits * tiles_x, t1 = (part + 1) * p.tiles_y / p.splits * tiles_x;  // its tiles
    const float mov_wf = p.mov_wf, mov_hf = p.mov_hf;
    const float *__restrict__ mdata = p.mov.data;
    const int mpitch = p.mov.pitch;
    const float *__restrict__ fdata = p.fix.data;
    const int fpitch = p.fix.pitch;

    // ---- the warp's points: coefficients, guard, slots
    SpanSlot *my_slots = ss.slots + warp * G;
    span_points<CGS_COST_ZNCC, G>(p, (task * NW + warp) * G, my_slots);
    __syncwarp();
    float2 A2[GP], C12[GP], D12[GP];
#pragma unroll
    for (int h = 0; h < GP; h++) {
        const SpanSlot &a = my_slots[2 * h], &b = my_slots[2 * h + 1];
        A2[h] = make_float2(a.A, b.A);
        C12[h] = make_float2(a.C1, b.C1);
        D12[h] = make_float2(a.D1, b.D1);
    }
    if (lane < GP) {
        const SpanSlot &a = my_slots[2 * lane], &b = my_slots[2 * lane + 1];
        ss.prow[warp * GP + lane] = PairRow{make_float2(a.B, b.B), make_float2(a.PQ, b.PQ), make_float2(a.C2, b.C2),
                                            make_float2(a.RS, b.RS), make_float2(a.D2, b.D2), make_float2(a.TU, b.TU)};
    }
    // FP64 task totals and overlap counts of the warp's points (shared memory)
    double *my_dtot = ss.dtot + warp * G * 5;
    int *my_cnt = ss.cnt + warp * G;
    double *my_band = ss.dband + warp * G * 5;
    for (int i = lane; i < G * 5; i += 32) my_dtot[i] = my_band[i] = 0.0;
    if (lane < G) my_cnt[lane] = 0;
    const float fshift = p.shifts[0], mshift = p.shifts[1];
    __syncthreads();  // every point's slot is written

    span_windows<1, G, NW, TX>(p, ss, t0, t1);
    __syncthreads();
    if (threadIdx.x == 0) expect_window<1, TX>(p, ss, t0);
    __syncthreads();
    issue_window<1, NW, TX>(p, ss, p.fix.data, t0);

    // ---- sweep
    float2 part_sum[GP][3];  // {sum m', sum m'^2, sum f'm'} of each pair of points
#pragma unroll
    for (int h = 0; h < GP; h++)
#pragma unroll
        for (int j = 0; j < 3; j++) part_sum[h][j] = make_float2(0.0f, 0.0f);
    InnerSpan *my_spans = ss.spans + warp * G * TH;
    RowRun *my_runs = ss.runs + warp * TH;
    const float2 magic2 = make_float2(kMagic, kMagic), minus1 = make_float2(-1.0f, -1.0f);
    // quad index from floor bits: bits(tx - pitch nfy) - kMagicBits = ix + pitch iy (exact below
    // 2^22; nfy = -floor y); global quad (ix, iy) at mqbase + 16 bits
    const uint64_t mqbase = reinterpret_cast<uint64_t>(p.mov_quad) - 16ull * (uint64_t)(uint32_t)kMagicBits;
    const float2 qpitch2 = make_float2(-(float)p.quad_pitch, -(float)p.quad_pitch);

    for (int t = t0; t < t1; t++, wit++) {
        const int tx = t % tiles_x, ty = t / tiles_x;
        const int x0 = tx * TW, y0 = ty * TH;
        const int x1 = min(x0 + TW, fw) - 1;
        if (tx == 0) {
            // the band's rows, every point of the warp: inner spans (their fixed-image sums from the
            // row prefix sums) and the band pixels, sampled by the reference's exact sequence;
            // entry i = g TH + r, lanes of one point reduce over its TH rows
            for (int k = 0; 32 * k < G * TH; k++) {
                const int i = lane + 32 * k;
                const bool act = i < G * TH;
                const int g = act ? i / TH : 0, r = i - g * TH;
                double s1 = 0.0, s2 = 0.0, sm = 0.0, smm = 0.0, sfm = 0.0;
                int n = 0;
                bool sure = true;
                const int y = y0 + r;
                const float yf = (float)y;
                RowSpans sp{0, 0, 0, 0};
                if (act) {
                    const SpanSlot &sl = my_slots[g];
                    if (y < fh && sl.valid) {
                        if (sl.ok) sp = row_spans(sl, yf, fw, mov_wf, mov_hf);
                        else sp.plen = fw;  // ill-conditioned: every pixel exact
                    }
                    my_spans[g * TH + r] = InnerSpan{sp.xa, sp.len};
                    n = sp.len;
                    if (sp.len > 0) {
                        const double2 *pr = p.fix_prefix + (int64_t)y * (fw + 1) + sp.xa;
                        const double2 a = pr[0], b = pr[sp.len];
                        s1 = b.x - a.x;
                        s2 = b.y - a.y;
                        sure = prefix_holds(s2, b.y);
                    }
                }
                for (uint32_t m = __ballot_sync(0xffffffffu, !sure); m; m &= m - 1u) {
                    const int l = __ffs(m) - 1;
                    const double2 t = row_sums<1>(p.fix, __shfl_sync(0xffffffffu, y, l), __shfl_sync(0xffffffffu, sp.xa, l),
                                                  __shfl_sync(0xffffffffu, sp.len, l));
                    if (lane == l) {
                        s1 = t.x;
                        s2 = t.y;
                    }
                }
                if (act) {
                    // band pixels: the outer span outside the inner one, [pa, e0) and [e1, pa + plen)
                    const SpanSlot &sl = my_slots[g];
                    const int e0 = sp.len > 0 ? sp.xa : sp.pa + sp.plen, e1 = sp.len > 0 ? sp.xa + sp.len : sp.pa + sp.plen;
                    const MapCoef kc{sl.A, sl.B, sl.P, sl.Q, sl.C1, sl.C2, sl.R, sl.S, sl.D1, sl.D2, sl.T, sl.U};
                    const float *frow_g = fdata + (int64_t)y * fpitch;
                    auto band = [&](int xs, int xe) {
                        for (int x = xs; x < xe; x++) {
                            float ex, ey;
                            exact_map(kc, (float)x, yf, ex, ey);
                            if (in_image(ey, ex, mov_wf, mov_hf)) {
                                const float m = bilinear_in(mdata, mpitch, ey, ex) - mshift;
                                const float f = frow_g[x];
                                const float fs = f - fshift;
                                s1 += (double)f;
                                s2 += (double)f * (double)f;
                                sm += (double)m;
                                smm += (double)m * (double)m;
                                sfm += (double)fs * (double)m;
                                n++;
                            }
                        }
                    };
                    band(sp.pa, e0);
                    band(e1, sp.pa + sp.plen);
                }
                // sum over the TH lanes of each point (TH is 8, 16 or 32); the moving sums exist only
                // where a band pixel was found inside, which is rare
                const bool found = __any_sync(0xffffffffu, smm != 0.0 || sm != 0.0);
                for (int o = 1; o < TH && o < 32; o <<= 1) {
                    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
                    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
                    n += __shfl_xor_sync(0xffffffffu, n, o);
                }
                if (found)
                    for (int o = 1; o < TH && o < 32; o <<= 1) {
                        sm += __shfl_xor_sync(0xffffffffu, sm, o);
                        smm += __shfl_xor_sync(0xffffffffu, smm, o);
                        sfm += __shfl_xor_sync(0xffffffffu, sfm, o);
                    }
                if (act && r == 0) {
                    double *d = my_band + g * 5;
                    d[0] += s1;
                    d[2] += s2;
                    if (found) {
                        d[1] += sm;
                        d[3] += smm;
                        d[4] += sfm;
                    }
                    my_cnt[g] += n;
                }
            }
            __syncwarp();
            if (lane < TH) {  // the rows' common inner run and the hull of the inner spans
                int ia = 0, ib = fw - 1, ua = 1 << 30, ub = -1;
#pragma unroll
                for (int g = 0; g < G; g++) {
                    const InnerSpan is = my_spans[g * TH + lane];
                    if (is.len > 0) {
                        ia = max(ia, is.xa);
                        ib = min(ib, is.xa + is.len - 1);
                        ua = min(ua, is.xa);
                        ub = max(ub, is.xa + is.len - 1);
                    } else {
                        ib = -1;  // a point without an inner span (or outside the grid): no common run
                    }
                }
                my_runs[lane] = RowRun{ia, ib, ua, ub};
            }
            __syncwarp();
        }
        // the tile's windows
        if (!mbar_wait_bounded(ss.bar, wit & 1u, kWaitLimitNs)) *ss.abort_flag = 1;
        const BlockWin *twin = ss.wins + t * TX;
        const float *sfix = reinterpret_cast<const float *>(ss.win);  // TH x TW
        const uint32_t wbase = smem_addr(ss.win + TH * TW / 4);
        const uint32_t szero = smem_addr(ss.win);

        // one row: fast samples of G points at the lane's columns; EDGE masks by the inner spans
        auto row = [&](int r, const RowRun run) {
            const int y = y0 + r;
            const float yf = (float)y;
            const float2 yf2 = make_float2(yf, yf);
            float2 byw[GP], byx[GP], byy[GP];
#pragma unroll
            for (int h = 0; h < GP; h++) {
                const PairRow pr = ss.prow[warp * GP + h];
                byw[h] = __ffma2_rn(pr.B, yf2, pr.PQ);
                byx[h] = __ffma2_rn(pr.C2, yf2, pr.RS);
                byy[h] = __ffma2_rn(pr.D2, yf2, pr.TU);
            }
            const float *frow = sfix + r * TW;
            // one block of 32 columns; EDGE: some column may lie outside a point's inner span;
            // SMEM: the block's window is in the stage
            auto column = [&](int c, auto edge_tag, auto smem_tag) {
                constexpr bool EDGE = decltype(edge_tag)::value;
                constexpr bool SMEM = decltype(smem_tag)::value;
                // shared address of window quad (ix, iy): wbase + 16 (off + (ix - x0) + pitch (iy - y0))
                uint32_t sbase = 0u;
                float2 pitch2 = qpitch2;
                if constexpr (SMEM) {
                    const uint2 rp = *reinterpret_cast<const uint2 *>(&twin[c].rel);
                    sbase = wbase + rp.x;
                    pitch2 = make_float2(__uint_as_float(rp.y), __uint_as_float(rp.y));
                }
                InnerSpan isp[G];
                if constexpr (EDGE) {
#pragma unroll
                    for (int g = 0; g < G; g++) isp[g] = my_spans[g * TH + r];
                }
                const int x = x0 + 32 * c + lane;
                const float f = frow[32 * c + lane];  // past the image's right edge: not copied, unused
                const float fs = f - fshift;
                const float2 fs2 = make_float2(fs, fs);
                const float xf = (float)x;
                const float2 xf2 = make_float2(xf, xf);
#pragma unroll
                for (int h = 0; h < GP; h++) {
                    // both points of the pair in each FP32x2 operation: map, floor (the product X / w
                    // added to 1.5 * 2^23 with one rounding down leaves floor(X / w) in the mantissa),
                    // its negative, fraction (X / w - floor, one rounding), quad index; the product is
                    // never rounded by itself, which saves two operations of twelve
                    const float2 w = __ffma2_rn(A2[h], xf2, byw[h]);
                    const float2 X = __ffma2_rn(C12[h], xf2, byx[h]);
                    const float2 Y = __ffma2_rn(D12[h], xf2, byy[h]);
                    const float2 rw = make_float2(rcp_approx(w.x), rcp_approx(w.y));
                    const float2 tx2 = __ffma2_rd(X, rw, magic2), ty2 = __ffma2_rd(Y, rw, magic2);
                    const float2 nfx2 = __ffma2_rn(tx2, minus1, magic2), nfy2 = __ffma2_rn(ty2, minus1, magic2);
                    const float2 ax2 = __ffma2_rn(X, rw, nfx2), ay2 = __ffma2_rn(Y, rw, nfy2);
                    const float2 qi = __ffma2_rn(nfy2, pitch2, tx2);
                    bool in0 = true, in1 = true;
                    if constexpr (EDGE) {
                        const InnerSpan a = isp[2 * h], b = isp[2 * h + 1];
                        in0 = (unsigned)(x - a.xa) < (unsigned)a.len;
                        in1 = (unsigned)(x - b.xa) < (unsigned)b.len;
                    }
                    uint32_t q0b = __float_as_uint(qi.x), q1b = __float_as_uint(qi.y);
                    if constexpr (EDGE) {
                        q0b = in0 ? q0b : (uint32_t)kMagicBits;
                        q1b = in1 ? q1b : (uint32_t)kMagicBits;
                    }
                    float4 q0, q1;
                    if constexpr (SMEM) {
                        uint32_t a0 = sbase + (q0b << 4), a1 = sbase + (q1b << 4);
                        if constexpr (EDGE) {
                            a0 = in0 ? a0 : szero;
                            a1 = in1 ? a1 : szero;
                        }
                        if constexpr (CHECK) {  // inside the block's window, else recorded and skipped
                            const BlockWin bw = twin[c];
                            const int ix0 = (int)(__float_as_uint(tx2.x) - (uint32_t)kMagicBits) - bw.x0;
                            const int iy0 = (int)(__float_as_uint(ty2.x) - (uint32_t)kMagicBits) - bw.y0;
                            const int ix1 = (int)(__float_as_uint(tx2.y) - (uint32_t)kMagicBits) - bw.x0;
                            const int iy1 = (int)(__float_as_uint(ty2.y) - (uint32_t)kMagicBits) - bw.y0;
                            const bool b0 = in0 && ((unsigned)ix0 >= (unsigned)bw.w || (unsigned)iy0 >= (unsigned)bw.h);
                            const bool b1 = in1 && ((unsigned)ix1 >= (unsigned)bw.w || (unsigned)iy1 >= (unsigned)bw.h);
                            if (b0 | b1) *ss.bounds_flag = 1;
                            a0 = b0 ? szero : a0;
                            a1 = b1 ? szero : a1;
                        }
                        // the stage is ready (its barrier was waited on above); volatile keeps the
                        // loads after that wait
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                     : "=f"(q0.x), "=f"(q0.y), "=f"(q0.z), "=f"(q0.w) : "r"(a0));
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                     : "=f"(q1.x), "=f"(q1.y), "=f"(q1.z), "=f"(q1.w) : "r"(a1));
                    } else {
                        if constexpr (CHECK) {  // inside the moving image, else recorded and skipped
                            const int ix0 = (int)(__float_as_uint(tx2.x) - (uint32_t)kMagicBits);
                            const int iy0 = (int)(__float_as_uint(ty2.x) - (uint32_t)kMagicBits);
                            const int ix1 = (int)(__float_as_uint(tx2.y) - (uint32_t)kMagicBits);
                            const int iy1 = (int)(__float_as_uint(ty2.y) - (uint32_t)kMagicBits);
                            const bool b0 = in0 && ((unsigned)ix0 >= (unsigned)p.mov.w || (unsigned)iy0 >= (unsigned)p.mov.h);
                            const bool b1 = in1 && ((unsigned)ix1 >= (unsigned)p.mov.w || (unsigned)iy1 >= (unsigned)p.mov.h);
                            if (b0 | b1) *ss.bounds_flag = 1;
                            q0b = b0 ? (uint32_t)kMagicBits : q0b;
                            q1b = b1 ? (uint32_t)kMagicBits : q1b;
                        }
                        q0 = __ldg(reinterpret_cast<const float4 *>(mqbase + 16ull * q0b));
                        q1 = __ldg(reinterpret_cast<const float4 *>(mqbase + 16ull * q1b));
                    }
                    // quad = the bilinear polynomial's coefficients {c00 - s_m, c10, c01, c11}:
                    // m' = (c00 - s_m + ax c10) + ay (c01 + ax c11)
                    const float u0 = fmaf(ax2.x, q0.y, q0.x), w0 = fmaf(ax2.x, q0.w, q0.z);
                    const float u1 = fmaf(ax2.y, q1.y, q1.x), w1 = fmaf(ax2.y, q1.w, q1.z);
                    float2 ms = make_float2(fmaf(ay2.x, w0, u0), fmaf(ay2.y, w1, u1));
                    float2 fm = fs2;
                    if constexpr (EDGE) {  // by selection: a NaN outside the overlap stays out of the sums
                        ms = make_float2(in0 ? ms.x : 0.0f, in1 ? ms.y : 0.0f);
                        fm = make_float2(in0 ? fs : 0.0f, in1 ? fs : 0.0f);
                    }
                    part_sum[h][0] = __fadd2_rn(part_sum[h][0], ms);
                    part_sum[h][1] = __ffma2_rn(ms, ms, part_sum[h][1]);
                    part_sum[h][2] = __ffma2_rn(fm, ms, part_sum[h][2]);
                }
            };
            auto block = [&](int c, auto edge_tag) {
                if (twin[c].w > 0) column(c, edge_tag, std::true_type{});
                else column(c, edge_tag, std::false_type{});
            };
            // blocks with any inner span: [cu0, cu1]; those inside every point's inner span,
            // [cf0, cf1], run unmasked
            const int cu0 = max(0, (run.ua - x0) >> 5), cu1 = min(TX - 1, (run.ub - x0) >> 5);
            int cf0 = cu1 + 1, cf1 = cu1;
            if (run.ia <= run.ib) {
                const int a = max(cu0, (run.ia - x0 + 31) >> 5), b = min(cu1, ((run.ib - x0 + 1) >> 5) - 1);
                if (a <= b) {
                    cf0 = a;
                    cf1 = b;
                }
            }
#pragma unroll 1
            for (int c = cu0; c < cf0; c++) block(c, std::true_type{});
            int c = cf0;
#pragma unroll 1
            for (; c + 1 <= cf1; c += 2) {  // two full blocks of the same kind as straight-line code
                const bool s0 = twin[c].w > 0, s1 = twin[c + 1].w > 0;
                if (s0 && s1) {
                    column(c, std::false_type{}, std::true_type{});
                    column(c + 1, std::false_type{}, std::true_type{});
                } else if (!s0 && !s1) {
                    column(c, std::false_type{}, std::false_type{});
                    column(c + 1, std::false_type{}, std::false_type{});
                } else {
                    block(c, std::false_type{});
                    block(c + 1, std::false_type{});
                }
            }
            if (c <= cf1) block(c, std::false_type{});
#pragma unroll 1
            for (int c2 = cf1 + 1; c2 <= cu1; c2++) block(c2, std::true_type{});
        };
        for (int r = 0; r < TH; r++) {
            if (y0 + r >= fh) break;
            const RowRun run = my_runs[r];
            if (run.ua > x1 || run.ub < x0) continue;  // no point samples this row of the tile
            row(r, run);
        }
        // end of a band of tiles: the band's warp sums into the FP64 task totals
        if (tx == tiles_x - 1) {
#pragma unroll
            for (int h = 0; h < GP; h++)
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    const int slot = j == 0 ? 1 : (j == 1 ? 3 : 4);  // sum m', sum m'^2, sum f'm'
                    const float s0 = warp_sum(part_sum[h][j].x), s1 = warp_sum(part_sum[h][j].y);
                    if (lane == 0) {
                        my_band[(2 * h) * 5 + slot] += (double)s0;
                        my_band[(2 * h + 1) * 5 + slot] += (double)s1;
                    }
                    part_sum[h][j] = make_float2(0.0f, 0.0f);
                }
            fold_band<G, NW>(p, task, ty, my_dtot, my_band);
        }
        const bool more = t + 1 < t1;
        if (threadIdx.x == 0 && more) expect_window<1, TX>(p, ss, t + 1);
        __syncthreads();  // every warp is done with the stage
        if (*ss.abort_flag) {  // a wait gave up: let the stage's copies land, within the same bound, before the CTA stops
            if (threadIdx.x == 0) mbar_wait_bounded(ss.bar, wit & 1u, kWaitLimitNs);
            return false;
        }
        if (more) issue_window<1, NW, TX>(p, ss, p.fix.data, t + 1);
    }

    if (!join_parts<G, NW, CHECK>(p, task, part, ss, my_dtot, my_cnt)) return true;

    // ---- per grid point: finalise, dump, argmin key (as the pixel-loop kernel)
    __syncwarp();
    unsigned long long kk = ~0ull;
    if (lane < G) {
        const SpanSlot &sl = my_slots[lane];
        const int n = my_cnt[lane];
        // the fixed-image sums were taken unshifted: sum f' = sum f - n s, sum f'^2 = sum f^2 -
        // 2 s sum f + n s^2 (FP64)
        const double s = (double)fshift, dn = (double)n;
        double a[5];
#pragma unroll
        for (int j = 0; j < 5; j++) a[j] = my_dtot[lane * 5 + j];
        const double f1 = a[0];
        a[0] = f1 - dn * s;
        a[2] = a[2] - 2.0 * s * f1 + dn * s * s;
        const float cost = zncc_cost(a, n, p);
        if (sl.valid) {
            if (p.costs) p.costs[sl.index] = cost;
            kk = make_key(cost, sl.index);
        }
    }
    kk = warp_min_u64(kk);
    if (lane == 0) ss.wbest[warp] = kk;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long b = ~0ull;
        for (int w = 0; w < NW; w++) b = ss.wbest[w] < b ? ss.wbest[w] : b;
        retire_tasks(p, b, 1u, false);
    }
    return true;
}

// The single-pair span kernel: persistent CTAs, tasks (or their parts) dealt round-robin.
template <int G, int NW, int TX, bool CHECK>
__global__ void __launch_bounds__(NW * 32, 1) span_kernel(const __grid_constant__ SearchParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    const SpanSmem ss = carve_span<G, NW>(smem, p.tile_h, TX, p.tiles_x * p.tiles_y, p.win_cap);
    if (threadIdx.x == 0) {
        mbar_init(ss.bar, 1);
        fence_mbar_init();
        *ss.abort_flag = 0;
        *ss.bounds_flag = 0;
    }
    __syncthreads();
    const uint32_t units = p.num_tasks * (uint32_t)p.splits;
    uint32_t wit = 0;
    for (uint32_t u = blockIdx.x; u < units; u += gridDim.x) {
        if (!run_span_task<G, NW, TX, CHECK>(p, u, ss, wit)) {
            if (threadIdx.x == 0) retire_parts(p, u, gridDim.x, units);
            return;
        }
    }
}

// Blocks [0, row_blocks) write the FP64 prefix sums of each staged fixed row, prefix[y (W + 1) +
// x] = {sum f, sum f^2} of pixels 0 .. x - 1 of row y (over the channels; one warp per row, a warp scan
// per 32 pixels carried in order, so the sums are the same in every run); the other blocks of
// the `nblocks` subtract the moving image's shift from every quad's constant term, so that the
// sweep's bilinear values are shifted already.
__device__ __forceinline__ void span_prep_body(const SpanPrepArgs &a, int block, int nblocks) {
    if (block >= a.row_blocks) {
        const float ms = a.shifts[1];
        const int64_t nthr = (int64_t)(nblocks - a.row_blocks) * blockDim.x;
        for (int64_t i = (int64_t)(block - a.row_blocks) * blockDim.x + threadIdx.x; i < a.nquads; i += nthr)
            a.quads[i].x -= ms;
        return;
    }
    const int row = (int)((block * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (row >= a.fh) return;
    const int fw = a.fw;
    const float *src = a.fix + (int64_t)row * a.fpitch;
    double2 *dst = a.prefix + (int64_t)row * (fw + 1);
    if (lane == 0) dst[0] = make_double2(0.0, 0.0);
    double c1 = 0.0, c2 = 0.0;
    for (int x0 = 0; x0 < fw; x0 += 32) {
        const int x = x0 + lane;
        double v = 0.0, v2 = 0.0;
        for (int ch = 0; x < fw && ch < a.channels; ch++) {
            const double u = (double)src[ch * a.fplane + x];
            v += u;
            v2 += u * u;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double t1 = __shfl_up_sync(0xffffffffu, v, o), t2 = __shfl_up_sync(0xffffffffu, v2, o);
            if (lane >= o) {
                v += t1;
                v2 += t2;
            }
        }
        if (x < fw) dst[x + 1] = make_double2(c1 + v, c2 + v2);
        c1 += __shfl_sync(0xffffffffu, v, 31);
        c2 += __shfl_sync(0xffffffffu, v2, 31);
    }
}

static __global__ void __launch_bounds__(256) span_prep_kernel(const SpanPrepArgs a) {
    span_prep_body(a, (int)blockIdx.x, (int)gridDim.x);
}

// The staging step of many pairs at once: pair blockIdx.y, its blocks blockIdx.x (gridDim.x
// exceeds every pair's row_blocks).
static __global__ void __launch_bounds__(256) span_prep_batch_kernel(const SpanPrepArgs *__restrict__ args) {
    span_prep_body(args[blockIdx.y], (int)blockIdx.x, (int)gridDim.x);
}

}  // namespace cgs
