// cgs_span_exact.cuh -- the span kernel of the costs that need the reference's samples bit for bit:
// averageAbsoluteDifference (SAD_AVG), calcSQD (SQD_REF), calcNCC (NCC_REF) and the joint-histogram MI,
// one or three channels.  Every sample is formed by the reference's operation sequence, as the
// per-sample kernel does; what changes is around it: the in/out decisions are taken per image row, the
// taps come from shared-memory windows and the quotients need no branch.
//
// Decisions, tiles, windows, stage: as in the zero-mean NCC span kernel (cgs_span.cuh).  A point's
// inner span lies at least 1.5 guard bands inside the moving image, and the guard bounds the distance
// between the real and the reference's coordinates, so every pixel of the inner span is inside for the
// reference; band pixels are decided and sampled in the span pass.  A point without a guard, or whose
// quotients could leave exact_quot2's range, has no spans: the whole warp samples all of its pixels
// with IEEE divisions (band_pixels).
//
// Sweep.  Lane l takes the columns x0 + 32 c + l of a tile, block c after block c and in each block
// the rows that have samples there (two ballots per block sort the rows into full, masked and none).
// A block's products A x, C1 x, D1 x are formed once for its rows and the rows' B y, C2 y, D2 y once per
// band (shared memory): three of 29 packed operations per sample and pair saved.  Two points per
// FP32x2 operation; with one pair per warp two rows run at once.  The map keeps the reference's order
// w = ((A x + B y) + P) - Q with each operation rounded; X and Y are formed with negated coefficients
// (the same bits, sign flipped), which the quotient step wants.  Floors and fractions are exact
// operations.  The quads hold the raw taps {v00, v01, v10, v11}.  The row weights carry a power of two,
// so samples come out scaled by it, the same bits: 2^-8 for the NCC-like costs, whose sums of squares
// then have the headroom of the reference's v / 255 without its division (the factor leaves in FP64 at
// the end), and B / 256 for MI, whose sample is then its bin after a clamp and a floor.
//
// What bounds it: the FP32 pipe.  A pair of points takes 26 packed operations (two pipe cycles each)
// and about 20 scalar ones per pixel and channel; the heavier of the two FP32 pipes is active on 72 % of
// cycles (SAD, 256 x 256).  39 instructions per 32 evaluations, of which 5 are register moves.  Whole
// calls: SAD 64 x 64, 4^8, 645 us against 839 on the per-sample kernel; calcNCC 203 x 157 3.86 ms against 6.2.
// Row after row instead of block after block 9 % slower.
//
// Three-channel MI runs here too (2.8 ms against 4.7 on the per-sample kernel for 301 x 211, 3^8); with
// one channel the guarded fast samples of cgs_span_mi.cuh are faster.
//
// MI counts.  Each warp keeps its points' (B + 1) x (B + 1) u32 histograms in shared memory (row = fixed
// bin, the last row and column for the marginals), filled with shared-memory atomics; the tile's fixed
// rows are the fixed image's bins times the row stride, in bytes.  The cost is formed by mi_from_hist,
// as in the per-sample kernel: equal counts give equal bits.
//
// Sums of the other costs.  Per lane and band of TH rows in FP32, then a warp sum into FP64 totals; the
// fixed image's sum of squares comes from the row prefix sums (or the pixels: prefix_holds).  SAD is
// formed in FP64, the NCC-like costs in FP32 from the rounded totals (finalize), so their special cases
// are the per-sample kernel's.  Costs do not depend on the order of the points or on how many share a
// launch.
#pragma once
#include "cgs_span.cuh"

namespace cgs {

// FP32 sums of a pair of points in the sweep: SAD {sum |d|}; SQD {sum d^2, sum m^2}; NCC {sum m^2, sum f m}.
template <int COST> struct SpanSums {
    static constexpr int value = COST == CGS_COST_SAD_AVG || COST == CGS_COST_MI ? 1 : 2;
};

// Shared memory of the exact span kernel: the span kernels' (carve_span), the rows' products B y, -C2 y,
// -D2 y of the warps' pairs, [NW][TH][G / 2], and the MI histograms, [NW * G][(B + 1)^2], before the
// window stage.
__host__ __device__ constexpr size_t span_exact_extra(int G, int NW, int TH, int mi_bins) {
    return (((size_t)NW * TH * (G / 2) * 24 + 15) & ~(size_t)15) +
           (mi_bins > 0 ? (((size_t)NW * G * (mi_bins + 1) * (mi_bins + 1) * 4 + 15) & ~(size_t)15) : 0);
}

// One (fixed f, moving m) sample, both scaled, into FP64 sums.
template <int COST>
__device__ __forceinline__ void accumulate64(double *a, float f, float m) {
    const float d = m - f;
    if constexpr (COST == CGS_COST_SAD_AVG) {
        a[0] += (double)fabsf(d);
    } else if constexpr (COST == CGS_COST_MI) {
    } else if constexpr (COST == CGS_COST_SQD_REF) {
        a[0] += (double)d * (double)d;
        a[1] += (double)m * (double)m;
    } else {
        a[0] += (double)m * (double)m;
        a[1] += (double)f * (double)m;
    }
}

// The band pixels of a row: the outer span outside the inner one, [pa, e0) and [e1, pe).
struct RowBand {
    int pa, e0, e1, pe;
    __device__ __forceinline__ explicit RowBand(const RowSpans &s)
        : pa(s.pa), e0(s.len > 0 ? s.xa : s.pa + s.plen), e1(s.len > 0 ? s.xa + s.len : s.pa + s.plen), pe(s.pa + s.plen) {}
    __device__ __forceinline__ bool many() const { return (e0 - pa) + (pe - e1) > kFewBand; }
};

// The samples of a point outside its inner spans: the reference's sequence, scaled by kS.
template <int COST, int C>
struct SpanSampler {
    static constexpr int NS = SpanSums<COST>::value;
    MapCoef kc;
    Plane mov, fix;
    float mw, mh, kS;
    uint32_t hist;  // shared address of the point's histogram
    int B;
    double a[NS] = {}, s2 = 0.0;  // the sums, sum f^2
    int n = 0;
    __device__ __forceinline__ SpanSampler(const SearchParams &p, const SpanSlot &sl, const uint32_t *h, float scale)
        : kc{sl.A, sl.B, sl.P, sl.Q, sl.C1, sl.C2, sl.R, sl.S, sl.D1, sl.D2, sl.T, sl.U}, mov(p.mov), fix(p.fix),
          mw(p.mov_wf), mh(p.mov_hf), kS(scale), hist(smem_addr(h)), B(p.mi_bins) {}
    __device__ __forceinline__ void add(int x, int y) {
        float ex, ey;
        exact_map(kc, (float)x, (float)y, ex, ey);
        if (!in_image(ey, ex, mw, mh)) return;
#pragma unroll
        for (int ch = 0; ch < C; ch++) {
            const float m = bilinear_in(mov.data + ch * mov.plane, mov.pitch, ey, ex);
            const float f = __ldg(fix.data + ch * fix.plane + (int64_t)y * fix.pitch + x);
            if constexpr (COST == CGS_COST_MI) red_shared_add1(hist + 4u * (uint32_t)(mi_bin(f, kS, B) * (B + 1) + mi_bin(m, kS, B)));
            else accumulate64<COST>(a, f * kS, m * kS);
            if constexpr (COST == CGS_COST_SQD_REF || COST == CGS_COST_NCC_REF) s2 += (double)f * (double)f;
        }
        n++;
    }
};

// What few bands of rows have: the band pixels of the rows from y0 of the warp's points, a few by the row's
// lane, many (a row along an edge of the moving image has nothing else) by the warp, and every pixel of
// the points without spans.  parts: a bit per 32 (point, row) entries that have band pixels.  A function
// of its own, which leaves the sweep its registers (SAD 256 x 256 7.01 ms against 7.15-7.25 inlined).  The
// multi-pair kernel, whose bodies share one register allocation, spills around such a call (8 % slower): it
// samples the same pixels in the span pass itself.
template <int COST, int C, int G>
__device__ __noinline__ void band_pixels(const SearchParams &p, const SpanSlot *slots, double *band, int *cnt, uint32_t *hist,
                                         float kS, int y0, uint32_t parts) {
    using Sampler = SpanSampler<COST, C>;
    const int lane = threadIdx.x & 31, TH = p.tile_h, fw = p.fix.w, fh = p.fix.h;
    const int hsize = (p.mi_bins + 1) * (p.mi_bins + 1);
    // the sums of groups of `width` lanes into their points' totals
    auto add = [&](int g, Sampler &s, int width, bool leader) {
        for (int o = 1; o < width; o <<= 1) {
            if constexpr (COST != CGS_COST_MI) {
                s.s2 += __shfl_xor_sync(0xffffffffu, s.s2, o);
#pragma unroll
                for (int j = 0; j < Sampler::NS; j++) s.a[j] += __shfl_xor_sync(0xffffffffu, s.a[j], o);
            }
            s.n += __shfl_xor_sync(0xffffffffu, s.n, o);
        }
        if (leader) {
            if constexpr (COST != CGS_COST_MI) {
                band[g * 5] += s.s2;
#pragma unroll
                for (int j = 0; j < Sampler::NS; j++) band[g * 5 + 1 + j] += s.a[j];
            }
            cnt[g] += s.n;
        }
        __syncwarp();
    };
    auto run = [&](int g, int ya, int ye, int xa, int xb, int xc, int xd) {  // pixels [xa, xb) and [xc, xd)
        Sampler s(p, slots[g], hist + g * hsize, kS);
        for (int y = ya; y < ye; y++) {
#pragma unroll (COST == CGS_COST_MI ? 2 : 4)
            for (int x = xa + lane; x < xb; x += 32) s.add(x, y);
            for (int x = xc + lane; x < xd; x += 32) s.add(x, y);
        }
        add(g, s, 32, lane == 0);
    };
    for (; parts; parts &= parts - 1u) {
        const int i = lane + 32 * (__ffs(parts) - 1);
        const bool act = i < G * TH;
        const int g = act ? i / TH : 0, y = y0 + i - g * TH;
        RowSpans sp{0, 0, 0, 0};
        if (act && y < fh && slots[g].valid && slots[g].ok) sp = row_spans(slots[g], (float)y, fw, p.mov_wf, p.mov_hf);
        const RowBand b(sp);
        Sampler s(p, slots[g], hist + g * hsize, kS);
        if (!b.many()) {
            for (int x = b.pa; x < b.e0; x++) s.add(x, y);
            for (int x = b.e1; x < b.pe; x++) s.add(x, y);
        }
        if (__any_sync(0xffffffffu, s.n > 0)) add(g, s, TH, act && i == g * TH);
        for (uint32_t m = __ballot_sync(0xffffffffu, b.many()); m; m &= m - 1u) {
            const int l = __ffs(m) - 1, yl = __shfl_sync(0xffffffffu, y, l);
            run(__shfl_sync(0xffffffffu, g, l), yl, yl + 1, __shfl_sync(0xffffffffu, b.pa, l),
                __shfl_sync(0xffffffffu, b.e0, l), __shfl_sync(0xffffffffu, b.e1, l), __shfl_sync(0xffffffffu, b.pe, l));
        }
    }
    for (int g = 0; g < G; g++)
        if (slots[g].valid && !slots[g].ok) run(g, y0, min(y0 + TH, fh), 0, fw, 0, 0);
}

// MULTI: a body of the multi-pair kernel.
template <int COST, int C, int G, int NW, int TX, bool CHECK, bool MULTI = false>
__device__ __forceinline__ bool run_span_exact_task(const SearchParams &p, uint32_t unit, const SpanSmem &ss,
                                                    uint32_t &wit) {
    static_assert(G % 2 == 0, "the span path pairs grid points");
    constexpr int GP = G / 2;
    constexpr int NB = GP == 1 ? 2 : 1;  // full rows at once
    constexpr int TW = 32 * TX;
    constexpr int NS = SpanSums<COST>::value;
    constexpr bool kMI = COST == CGS_COST_MI;
    constexpr bool kFix = COST == CGS_COST_SQD_REF || COST == CGS_COST_NCC_REF;  // the cost needs sum f^2
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int fw = p.fix.w, fh = p.fix.h;
    const int TH = p.tile_h;
    const int tiles_x = p.tiles_x;
    const uint32_t task = unit / (uint32_t)p.splits;
    const int part = (int)(unit - task * (uint32_t)p.splits);
    const int t0 = part * p.tiles_y / p.splits * tiles_x, t1 = (part + 1) * p.tiles_y / p.splits * tiles_x;  // its tiles
    const float mov_wf = p.mov_wf, mov_hf = p.mov_hf;
    const int B = p.mi_bins, hstride = B + 1, hsize = hstride * hstride;
    // the samples' scale (a power of two)
    const float kS = kMI ? (float)B * (1.0f / 256.0f) : COST == CGS_COST_SAD_AVG ? 1.0f : 0x1p-8f;

    // ---- the warp's points
    SpanSlot *my_slots = ss.slots + warp * G;
    span_points<COST, G, true>(p, (task * NW + warp) * G, my_slots);
    __syncwarp();
    bool nospan = false;  // some point of the warp has no spans
#pragma unroll
    for (int g = 0; g < G; g++) nospan |= my_slots[g].valid && !my_slots[g].ok;
    float2 *my_rows = ss.rowtab + (size_t)warp * TH * GP * 3;  // [TH][GP]{B y, -C2 y, -D2 y}
    uint32_t *my_hist = ss.hist + (size_t)warp * G * hsize;
    double *my_dtot = ss.dtot + warp * G * 5;  // {sum f^2, the sweep's NS sums} per point, stride 5
    double *my_band = ss.dband + warp * G * 5;  // of the current band
    int *my_cnt = ss.cnt + warp * G;
    if constexpr (kMI) {
        for (int i = lane; i < G * hsize; i += 32) my_hist[i] = 0u;
    } else {
        for (int i = lane; i < G * 5; i += 32) my_dtot[i] = my_band[i] = 0.0;
    }
    if (lane < G) my_cnt[lane] = 0;
    __syncthreads();  // every point's slot is written

    // the tile's fixed rows: the staged image, or MI's plane of bins
    const float *fsrc = kMI ? p.span_rows : p.fix.data;
    span_windows<C, G, NW, TX>(p, ss, t0, t1);
    __syncthreads();
    if (threadIdx.x == 0) expect_window<C, TX>(p, ss, t0);
    __syncthreads();
    issue_window<C, NW, TX>(p, ss, fsrc, t0);

    // one sample of point g at (x, y) by the reference's sequence, into a (and f^2 into s2) or the
    // histogram if inside
    auto exact_sample = [&](int g, int x, int y, double *a, double &s2) -> int {
        const SpanSlot &sl = my_slots[g];
        const MapCoef kc{sl.A, sl.B, sl.P, sl.Q, sl.C1, sl.C2, sl.R, sl.S, sl.D1, sl.D2, sl.T, sl.U};
        float ex, ey;
        exact_map(kc, (float)x, (float)y, ex, ey);
        if (!in_image(ey, ex, mov_wf, mov_hf)) return 0;
#pragma unroll
        for (int ch = 0; ch < C; ch++) {
            const float m = bilinear_in(p.mov.data + ch * p.mov.plane, p.mov.pitch, ey, ex);
            const float f = p.fix.data[ch * p.fix.plane + (int64_t)y * p.fix.pitch + x];
            if constexpr (kMI)
                red_shared_add1(smem_addr(my_hist + g * hsize + mi_bin(f, kS, B) * hstride + mi_bin(m, kS, B)));
            else
                accumulate64<COST>(a, f * kS, m * kS);
            if constexpr (kFix) s2 += (double)f * (double)f;
        }
        return 1;
    };
    // adds the lanes' FP64 sums of point g (lanes of one group of `width`) into its totals
    auto add_totals = [&](int g, bool leader, int width, double *a, double s2, int n, bool moving) {
        for (int o = 1; o < width; o <<= 1) {
            if constexpr (kFix) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            n += __shfl_xor_sync(0xffffffffu, n, o);
        }
        if (!kMI && moving)
            for (int o = 1; o < width; o <<= 1)
#pragma unroll
                for (int j = 0; j < NS; j++) a[j] += __shfl_xor_sync(0xffffffffu, a[j], o);
        if (leader) {
            double *d = my_band + g * 5;
            if constexpr (kFix) d[0] += s2;
            if (!kMI && moving)
#pragma unroll
                for (int j = 0; j < NS; j++) d[1 + j] += a[j];
            my_cnt[g] += n;
        }
    };
    // every pixel of the band's rows for the points without spans, all lanes over the columns
    auto no_span_rows = [&](int y0, int y1) {
        for (int g = 0; g < G; g++) {
            const SpanSlot &sl = my_slots[g];
            if (!sl.valid || sl.ok) continue;
            double a[NS] = {}, s2 = 0.0;
            int n = 0;
            for (int y = y0; y < y1; y++)
                for (int x = lane; x < fw; x += 32) n += exact_sample(g, x, y, a, s2);
            add_totals(g, lane == 0, 32, a, s2, n, true);
            __syncwarp();
        }
    };

    // ---- sweep.  The points' coefficients,
    // w = ((A x + By) + P) + nQ, -X = ((nC1 x + nC2 y) + nR) + S, -Y alike,
    // and the sums are set at the start of a band, after its span pass, which then has their registers (the
    // multi-pair kernel, where that spills: once)
    float2 P2[GP], nQ2[GP], nR2[GP], S2[GP], nT2[GP], U2[GP];
    float2 acc[GP][NS];
    auto set_points = [&]() {
#pragma unroll
        for (int h = 0; h < GP; h++) {
            const SpanSlot &a = my_slots[2 * h], &b = my_slots[2 * h + 1];
            P2[h] = make_float2(a.P, b.P);
            nQ2[h] = make_float2(-a.Q, -b.Q);
            nR2[h] = make_float2(-a.R, -b.R);
            S2[h] = make_float2(a.S, b.S);
            nT2[h] = make_float2(-a.T, -b.T);
            U2[h] = make_float2(a.U, b.U);
#pragma unroll
            for (int j = 0; j < NS; j++) acc[h][j] = make_float2(0.0f, 0.0f);
        }
    };
    if constexpr (MULTI) set_points();
    InnerSpan *my_spans = ss.spans + warp * G * TH;
    RowRun *my_runs = ss.runs + warp * TH;
    const float2 magic2 = make_float2(kMagic, kMagic), minus1 = make_float2(-1.0f, -1.0f);
    const float2 one2 = make_float2(1.0f, 1.0f), s2c = make_float2(kS, kS);
    // -0, not known to the compiler: a product is a multiply-add of -0 (the same bits), because the
    // assembler contracts a packed multiplication into the packed addition that consumes it, rounding
    // modifiers notwithstanding (seen on CUDA 12.9; scalar ones are left alone)
    const float nzero = __uint_as_float(0x80000000u | ((uint32_t)p.dims >> 8));
    const float2 nzero2 = make_float2(nzero, nzero);
    const float2 nsc = make_float2(-kS, -kS), smagic2 = make_float2(kS * kMagic, kS * kMagic);
    const uint64_t mqbase = reinterpret_cast<uint64_t>(p.mov_quad) - 16ull * (uint64_t)(uint32_t)kMagicBits;
    const float ikS = 1.0f / kS;  // exact
    const uint64_t qplane = 16ull * (uint64_t)p.quad_plane;
    // MI: histogram address of (fixed bin, moving bin bits): 4 bits + the fixed bin's byte offset + hbase
    const uint32_t hbase = smem_addr(my_hist) - 4u * (uint32_t)kMagicBits, hpoint = 4u * (uint32_t)hsize;
    const float bin_max = (float)(B - 1);

    for (int t = t0; t < t1; t++, wit++) {
        const int tx = t % tiles_x, ty = t / tiles_x;
        const int x0 = tx * TW, y0 = ty * TH;
        const int x1 = min(x0 + TW, fw) - 1;
        if (tx == 0) {
            // the band's rows: spans, the fixed sums of the inner ones, the band pixels
            uint32_t parts = 0u;  // entries with band pixels
            for (int k = 0; 32 * k < G * TH; k++) {
                const int i = lane + 32 * k;
                const bool act = i < G * TH;
                const int g = act ? i / TH : 0, r = i - g * TH, y = y0 + r;
                RowSpans sp{0, 0, 0, 0};
                double s2 = 0.0;
                bool sure = true;
                if (act) {
                    const SpanSlot &sl = my_slots[g];
                    if (y < fh && sl.valid && sl.ok) sp = row_spans(sl, (float)y, fw, mov_wf, mov_hf);
                    my_spans[g * TH + r] = InnerSpan{sp.xa, sp.len};
                    if constexpr (kFix) {
                        if (sp.len > 0) {
                            const double2 *pr = p.fix_prefix + (int64_t)y * (fw + 1) + sp.xa;
                            const double to = pr[sp.len].y;
                            s2 = to - pr[0].y;
                            sure = prefix_holds(s2, to);
                        }
                    }
                }
                parts |= (__any_sync(0xffffffffu, sp.plen > sp.len) ? 1u : 0u) << k;
                if constexpr (kFix) {
                    for (uint32_t m = __ballot_sync(0xffffffffu, !sure); m; m &= m - 1u) {
                        const int l = __ffs(m) - 1;
                        const double t = row_sums<C>(p.fix, __shfl_sync(0xffffffffu, y, l), __shfl_sync(0xffffffffu, sp.xa, l),
                                                     __shfl_sync(0xffffffffu, sp.len, l)).y;
                        if (lane == l) s2 = t;
                    }
                }
                if constexpr (MULTI) {
                    double a[NS] = {};
                    int n = sp.len;
                    // band pixels: the outer span outside the inner one, [pa, e0) and [e1, pe).  First every lane
                    // its row's, if a few; then, row after row, the warp those of a row with many (one along an
                    // edge of the moving image has nothing else)
                    const int pe = sp.pa + sp.plen, e0 = sp.len > 0 ? sp.xa : pe, e1 = sp.len > 0 ? sp.xa + sp.len : pe;
                    const bool many = (e0 - sp.pa) + (pe - e1) > kFewBand;
                    uint32_t rows = __ballot_sync(0xffffffffu, many);
                    int gc = g, yc = y, xa = sp.pa, xb = many ? sp.pa : e0, xc = e1, xd = many ? e1 : pe, step = 1, width = TH;
                    bool first = act && r == 0;
                    for (;;) {
                        int nb = 0;
                        for (int x = xa; x < xb; x += step) nb += exact_sample(gc, x, yc, a, s2);
                        for (int x = xc; x < xd; x += step) nb += exact_sample(gc, x, yc, a, s2);
                        add_totals(gc, first, width, a, s2, n + nb, __any_sync(0xffffffffu, nb > 0));
                        if (rows == 0u) break;
                        const int l = __ffs(rows) - 1;
                        rows &= rows - 1u;
                        gc = __shfl_sync(0xffffffffu, g, l);
                        yc = __shfl_sync(0xffffffffu, y, l);
                        xa = __shfl_sync(0xffffffffu, sp.pa, l) + lane;
                        xb = __shfl_sync(0xffffffffu, e0, l);
                        xc = __shfl_sync(0xffffffffu, e1, l) + lane;
                        xd = __shfl_sync(0xffffffffu, pe, l);
                        step = width = 32;
                        first = lane == 0;
                        n = 0;
                        s2 = 0.0;
#pragma unroll
                        for (int j = 0; j < NS; j++) a[j] = 0.0;
                        __syncwarp();
                    }
                } else {
                    int n = sp.len;
                    for (int o = 1; o < TH; o <<= 1) {
                        if constexpr (kFix) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
                        n += __shfl_xor_sync(0xffffffffu, n, o);
                    }
                    if (act && r == 0) {
                        if constexpr (kFix) my_band[g * 5] += s2;
                        my_cnt[g] += n;
                    }
                }
            }
            __syncwarp();
            if constexpr (MULTI) {
                if (nospan) no_span_rows(y0, min(y0 + TH, fh));
            } else if (parts || nospan) {
                band_pixels<COST, C, G>(p, my_slots, my_band, my_cnt, my_hist, kS, y0, parts);
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
                        ib = -1;
                    }
                }
                my_runs[lane] = RowRun{ia, ib, ua, ub};
            }
            for (int i = lane; i < TH * GP; i += 32) {  // the rows' products
                const int r = i / GP, h = i - r * GP;
                const SpanSlot &a = my_slots[2 * h], &b = my_slots[2 * h + 1];
                const float yf = (float)(y0 + r);
                float2 *d = my_rows + i * 3;
                d[0] = make_float2(xm(a.B, yf), xm(b.B, yf));
                d[1] = make_float2(-xm(a.C2, yf), -xm(b.C2, yf));
                d[2] = make_float2(-xm(a.D2, yf), -xm(b.D2, yf));
            }
            __syncwarp();
            if constexpr (!MULTI) set_points();
        }
        if (!mbar_wait_bounded(ss.bar, wit & 1u, kWaitLimitNs)) *ss.abort_flag = 1;
        const BlockWin *twin = ss.wins + t * TX;
        const float *sfix = reinterpret_cast<const float *>(ss.win);  // C x TH x TW
        const uint32_t wbase = smem_addr(ss.win + C * TH * TW / 4);
        const uint32_t szero = smem_addr(ss.win);

        // this lane's row of the band (lanes past it: none)
        const RowRun lrun = lane < TH && y0 + lane < fh ? my_runs[lane] : RowRun{1, 0, 1 << 30, -1};
#pragma unroll 1
        for (int c = 0; c < TX; c++) {
            const int xb = x0 + 32 * c;
            // the rows with samples in the block, and those where the block lies in every point's inner span
            uint32_t any = __ballot_sync(0xffffffffu, lrun.ua <= xb + 31 && lrun.ub >= xb);
            const uint32_t full = __ballot_sync(0xffffffffu, lrun.ia <= xb && lrun.ib >= xb + 31);
            if (any == 0u) continue;
            const bool in_stage = twin[c].w > 0;
            const int x = xb + lane;
            const float xf = (float)x;
            const float2 xf2 = make_float2(xf, xf);
            float2 ax0[GP], cx0[GP], dx0[GP];  // A x, -C1 x, -D1 x
#pragma unroll
            for (int h = 0; h < GP; h++) {
                const SpanSlot &a = my_slots[2 * h], &b = my_slots[2 * h + 1];
                ax0[h] = __ffma2_rn(make_float2(a.A, b.A), xf2, nzero2);
                cx0[h] = __ffma2_rn(make_float2(-a.C1, -b.C1), xf2, nzero2);
                dx0[h] = __ffma2_rn(make_float2(-a.D1, -b.D1), xf2, nzero2);
            }
            uint32_t sbase = 0u, wplane = 0u;
            float pitch;
            if (in_stage) {
                // shared address of window quad (ix, iy): wbase + 16 (off + (ix - x0) + pitch (iy - y0))
                sbase = wbase + twin[c].rel;
                pitch = twin[c].pitchf * ikS;
                wplane = 16u * (uint32_t)(twin[c].pitch * twin[c].h);
            } else {
                pitch = -(float)p.quad_pitch * ikS;
            }
            const float2 pitch2 = make_float2(pitch, pitch);
            const float *fcol = sfix + 32 * c + lane;

            // NR rows from row r; EDGE: some column may lie outside a point's inner span; SMEM: the
            // block's window is in the stage
            auto rows = [&](int r, auto nr_tag, auto edge_tag, auto smem_tag) {
                constexpr int NR = decltype(nr_tag)::value;
                constexpr bool EDGE = decltype(edge_tag)::value;
                constexpr bool SMEM = decltype(smem_tag)::value;
                float f[NR][C];
#pragma unroll
                for (int k = 0; k < NR; k++)
#pragma unroll
                    for (int ch = 0; ch < C; ch++) {
                        f[k][ch] = fcol[(ch * TH + r + k) * TW];
                        if constexpr (kFix) f[k][ch] *= 0x1p-8f;
                    }
#pragma unroll
                for (int kh = 0; kh < NR * GP; kh++) {
                    const int k = kh / GP, h = kh - k * GP;
                    const float2 *rt = my_rows + ((r + k) * GP + h) * 3;
                    const float2 w = __fadd2_rn(__fadd2_rn(__fadd2_rn(ax0[h], rt[0]), P2[h]), nQ2[h]);
                    const float2 nX = __fadd2_rn(__fadd2_rn(__fadd2_rn(cx0[h], rt[1]), nR2[h]), S2[h]);
                    const float2 nY = __fadd2_rn(__fadd2_rn(__fadd2_rn(dx0[h], rt[2]), nT2[h]), U2[h]);
                    float2 ex, ey;
                    exact_quot2(w, nX, nY, ex, ey);
                    // floor (round-down add of 1.5 * 2^23 leaves it in the mantissa), fractions a and 1 - a
                    // (exact, and rounded as the reference's 1 - a), the y weights scaled by kS
                    const float2 tx2 = __fadd2_rd(ex, magic2), ty2 = __fadd2_rd(ey, magic2);
                    const float2 nfx2 = __ffma2_rn(tx2, minus1, magic2), nfy2 = __ffma2_rn(ty2, nsc, smagic2);
                    const float2 ax = __fadd2_rn(ex, nfx2), ay = __ffma2_rn(ey, s2c, nfy2);
                    const float2 ox = __ffma2_rn(ax, minus1, one2), oy = __ffma2_rn(ay, minus1, s2c);
                    const float2 qi = __ffma2_rn(nfy2, pitch2, tx2);
                    bool in0 = true, in1 = true;
                    if constexpr (EDGE) {
                        const InnerSpan a = my_spans[2 * h * TH + r + k], b = my_spans[(2 * h + 1) * TH + r + k];
                        in0 = (unsigned)(x - a.xa) < (unsigned)a.len;
                        in1 = (unsigned)(x - b.xa) < (unsigned)b.len;
                    }
                    uint32_t q0b = __float_as_uint(qi.x), q1b = __float_as_uint(qi.y);
                    if constexpr (EDGE) {
                        q0b = in0 ? q0b : (uint32_t)kMagicBits;
                        q1b = in1 ? q1b : (uint32_t)kMagicBits;
                    }
                    uint32_t a0 = 0u, a1 = 0u;
                    if constexpr (SMEM) {
                        a0 = sbase + (q0b << 4);
                        a1 = sbase + (q1b << 4);
                        if constexpr (EDGE) {
                            a0 = in0 ? a0 : szero;
                            a1 = in1 ? a1 : szero;
                        }
                    }
                    if constexpr (CHECK) {  // inside the block's window or the image, else recorded and skipped
                        const BlockWin bw = twin[c];
                        const int wx = SMEM ? bw.x0 : 0, wy = SMEM ? bw.y0 : 0;
                        const unsigned ww = SMEM ? bw.w : p.mov.w, wh = SMEM ? bw.h : p.mov.h;
                        const int ix0 = (int)(__float_as_uint(tx2.x) - (uint32_t)kMagicBits) - wx;
                        const int iy0 = (int)(__float_as_uint(ty2.x) - (uint32_t)kMagicBits) - wy;
                        const int ix1 = (int)(__float_as_uint(tx2.y) - (uint32_t)kMagicBits) - wx;
                        const int iy1 = (int)(__float_as_uint(ty2.y) - (uint32_t)kMagicBits) - wy;
                        const bool b0 = in0 && ((unsigned)ix0 >= ww || (unsigned)iy0 >= wh);
                        const bool b1 = in1 && ((unsigned)ix1 >= ww || (unsigned)iy1 >= wh);
                        if (b0 | b1) *ss.bounds_flag = 1;
                        a0 = b0 ? szero : a0;
                        a1 = b1 ? szero : a1;
                        q0b = b0 ? (uint32_t)kMagicBits : q0b;
                        q1b = b1 ? (uint32_t)kMagicBits : q1b;
                    }
#pragma unroll
                    for (int ch = 0; ch < C; ch++) {
                        float4 q0, q1;
                        if constexpr (SMEM) {
                            // a masked or skipped sample reads the stage's start, whatever the plane
                            const uint32_t o = ch * wplane;
                            const uint32_t b0 = (EDGE || CHECK) && C > 1 && a0 == szero ? szero : a0 + o;
                            const uint32_t b1 = (EDGE || CHECK) && C > 1 && a1 == szero ? szero : a1 + o;
                            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                         : "=f"(q0.x), "=f"(q0.y), "=f"(q0.z), "=f"(q0.w) : "r"(b0));
                            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                         : "=f"(q1.x), "=f"(q1.y), "=f"(q1.z), "=f"(q1.w) : "r"(b1));
                        } else {
                            q0 = __ldg(reinterpret_cast<const float4 *>(mqbase + ch * qplane + 16ull * q0b));
                            q1 = __ldg(reinterpret_cast<const float4 *>(mqbase + ch * qplane + 16ull * q1b));
                        }
                        // valueAt_bilinear's order: (1 - ay)((1 - ax) v00 + ax v01) + ay((1 - ax) v10 + ax v11)
                        const float t0 = xa(xm(ox.x, q0.x), xm(ax.x, q0.y)), b0v = xa(xm(ox.x, q0.z), xm(ax.x, q0.w));
                        const float t1 = xa(xm(ox.y, q1.x), xm(ax.y, q1.y)), b1v = xa(xm(ox.y, q1.z), xm(ax.y, q1.w));
                        float2 m = make_float2(xa(xm(oy.x, t0), xm(ay.x, b0v)), xa(xm(oy.y, t1), xm(ay.y, b1v)));
                        if constexpr (kMI) {
                            // m = v B / 256: clamped to [0, B - 1] and floored, the reference's bin
                            m = make_float2(fminf(fmaxf(m.x, 0.0f), bin_max), fminf(fmaxf(m.y, 0.0f), bin_max));
                            const float2 b2 = __fadd2_rd(m, magic2);
                            const uint32_t hf = hbase + __float_as_uint(f[k][ch]);
                            if (in0) red_shared_add1(hf + (2 * h) * hpoint + 4u * __float_as_uint(b2.x));
                            if (in1) red_shared_add1(hf + (2 * h + 1) * hpoint + 4u * __float_as_uint(b2.y));
                        } else {
                            float2 fm = make_float2(f[k][ch], f[k][ch]);
                            if constexpr (EDGE) {  // by selection: a NaN outside the overlap stays out of the sums
                                m = make_float2(in0 ? m.x : 0.0f, in1 ? m.y : 0.0f);
                                fm = make_float2(in0 ? fm.x : 0.0f, in1 ? fm.y : 0.0f);
                            }
                            if constexpr (COST == CGS_COST_SAD_AVG) {
                                const float2 d = __ffma2_rn(fm, minus1, m);
                                acc[h][0].x += fabsf(d.x);
                                acc[h][0].y += fabsf(d.y);
                            } else if constexpr (COST == CGS_COST_SQD_REF) {
                                const float2 d = __ffma2_rn(fm, minus1, m);
                                acc[h][0] = __ffma2_rn(d, d, acc[h][0]);
                                acc[h][1] = __ffma2_rn(m, m, acc[h][1]);
                            } else {
                                acc[h][0] = __ffma2_rn(m, m, acc[h][0]);
                                acc[h][1] = __ffma2_rn(fm, m, acc[h][1]);
                            }
                        }
                    }
                }
            };
            auto block = [&](auto smem_tag) {
                using One = std::integral_constant<int, 1>;
                using Many = std::integral_constant<int, NB>;
#pragma unroll 1
                while (any) {
                    const int r = __ffs(any) - 1;
                    if constexpr (NB == 2) {
                        if (((full >> r) & 3u) == 3u) {
                            rows(r, Many{}, std::false_type{}, smem_tag);
                            any &= ~(3u << r);
                            continue;
                        }
                    }
                    if ((full >> r) & 1u) rows(r, One{}, std::false_type{}, smem_tag);
                    else rows(r, One{}, std::true_type{}, smem_tag);
                    any &= any - 1u;
                }
            };
            if (in_stage) block(std::true_type{});
            else block(std::false_type{});
        }
        // end of a band of tiles: the band's warp sums into the FP64 totals
        if (!kMI && tx == tiles_x - 1) {
#pragma unroll
            for (int h = 0; h < GP; h++)
#pragma unroll
                for (int j = 0; j < NS; j++) {
                    const float s0 = warp_sum(acc[h][j].x), s1 = warp_sum(acc[h][j].y);
                    if (lane == 0) {
                        my_band[(2 * h) * 5 + 1 + j] += (double)s0;
                        my_band[(2 * h + 1) * 5 + 1 + j] += (double)s1;
                    }
                    if constexpr (MULTI) acc[h][j] = make_float2(0.0f, 0.0f);
                }
            fold_band<G, NW>(p, task, ty, my_dtot, my_band);
        }
        const bool more = t + 1 < t1;
        if (threadIdx.x == 0 && more) expect_window<C, TX>(p, ss, t + 1);
        __syncthreads();  // every warp is done with the stage
        if (*ss.abort_flag) {
            if (threadIdx.x == 0) mbar_wait_bounded(ss.bar, wit & 1u, kWaitLimitNs);
            return false;
        }
        if (more) issue_window<C, NW, TX>(p, ss, fsrc, t + 1);
    }

    if (!join_parts<G, NW, CHECK>(p, task, part, ss, my_dtot, my_cnt)) return true;  // MI: never split

    // ---- per grid point: the cost from the totals or the counts, dump, argmin key
    __syncwarp();
    unsigned long long kk = ~0ull;
    float cost = 0.0f;
    if constexpr (kMI) {
#pragma unroll
        for (int g = 0; g < G; g++) {
            const float c = mi_from_hist(my_hist + g * hsize, my_cnt[g] * C, B, hstride, p);
            if (lane == g) cost = c;
            __syncwarp();
        }
    } else if (lane < G) {
        const int n = my_cnt[lane] * C;
        const double *d = my_dtot + lane * 5;
        constexpr double k2 = (256.0 / 255.0) * (256.0 / 255.0);
        float a[3] = {0.0f, 0.0f, 0.0f};
        if constexpr (COST == CGS_COST_SQD_REF) {
            a[0] = (float)(d[1] * k2);
            a[1] = (float)(d[2] * k2);
            a[2] = (float)(d[0] * (1.0 / 65025.0));
        } else {
            a[0] = (float)(d[0] * (1.0 / 65025.0));
            a[1] = (float)(d[1] * k2);
            a[2] = (float)(d[2] * k2);
        }
        // 0 / 0 is NaN, as in the reference
        if constexpr (COST == CGS_COST_SAD_AVG) {
            // a sum beyond FP32 is infinite, as the reference's and the per-sample kernel's
            const double sum = (double)(float)d[1];
            cost = (float)((isinf(sum) ? sum : d[1]) / (double)n);
        } else {
            cost = finalize<COST>(a, n, p);
        }
    }
    if (lane < G) {
        const SpanSlot &sl = my_slots[lane];
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

// The single-pair kernel: persistent CTAs, tasks (or their parts) dealt round-robin.
template <int COST, int C, int G, int NW, int TX, bool CHECK>
__global__ void __launch_bounds__(NW * 32, 1) span_exact_kernel(const __grid_constant__ SearchParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    const SpanSmem ss = carve_span<G, NW>(smem, p.tile_h, TX, p.tiles_x * p.tiles_y, p.win_cap, true,
                                          COST == CGS_COST_MI ? p.mi_bins : 0);
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
        if (!run_span_exact_task<COST, C, G, NW, TX, CHECK>(p, u, ss, wit)) {
            if (threadIdx.x == 0) retire_parts(p, u, gridDim.x, units);
            return;
        }
    }
}

}  // namespace cgs
