// zim_tiles.cuh -- per-tile / per-pixel device code shared by the plain
// per-pair kernels and the persistent batch kernels, so both paths run the
// same arithmetic (bit-identical results).  Every multiply-add that matters
// is an explicit fmaf, so the results do not depend on a translation unit's
// contraction flags.
//
// Reference: PhaseShiftGrayCode3D/src/JSLAB_PhaseShiftDecoder_V2.cpp:18-182
// (pre-blur + decode body), JSLAB_PhaseEpipolarReconstructor_V2.cpp:368-395
// (setData remap), :933-1006 (stereoMatch), :405-461 (median + reprojection),
// :79-195 (pixel Gaussian, radius outlier filter).
#pragma once

#include <cmath>

#include "zim_internal.cuh"

namespace zt {

// ---------------------------------------------------------------- decode ----

constexpr int DX = 32, DY = 8;  // source-image tile of the batch's post-smooth queue

struct DecodeParams {
    int rows, cols, enc, n_ps;
    int shift[4];
    int fbase[4];      // first frame of each phase-shift frequency
    float sinv[64];    // sin(2 pi k / N) per frame (reference LUT order)
    float cosv[64];
    float w2d[9];      // pre-blur weights k_a * k_b
    float thr;
    int avg3;
    // heterodyne (integer fringe counts)
    int f0, f1, f2, f12, f23, f1_gt_f2;
    float f0_f12, f1_f23, f2_f23, inv_f12, inv_f23, inv_f1, inv_f2;
    // hierarchical
    int iratio[4];
    float fratio[4];
    // Gray code
    int gray_bits, gray_base, complementary;
    // HDR least squares (JSLAB_HDRPhaseFit.h:10-61)
    int hdr;
    float hdr_sat, hdr_min_amp;
};

inline void decode_params(const zim_decode_config* c, int rows, int cols, DecodeParams& p) {
    p = DecodeParams{};
    p.rows = rows;
    p.cols = cols;
    p.enc = c->encoding;
    p.n_ps = c->encoding == ZIM_ENC_HETERODYNE3 ? 3 : (c->encoding == ZIM_ENC_HIERARCHICAL ? c->n_freq : 1);
    int f = 0;
    for (int i = 0; i < p.n_ps; i++) {
        p.shift[i] = c->shift_num[i];
        p.fbase[i] = f;
        for (int k = 0; k < c->shift_num[i]; k++, f++) {
            // sin(2.0 * PI * k / inum) in double, as the reference builds its LUT
            p.sinv[f] = (float)std::sin(2.0 * 3.14159265358979323846 * k / c->shift_num[i]);
            p.cosv[f] = (float)std::cos(2.0 * 3.14159265358979323846 * k / c->shift_num[i]);
        }
    }
    double kb[3];
    if (c->preblur_sigma <= 0) { kb[0] = 0.25; kb[1] = 0.5; kb[2] = 0.25; }
    else {
        double t = std::exp(-0.5 / (c->preblur_sigma * c->preblur_sigma));
        double mul = 1.0 / (2.0 * t + 1.0);
        kb[0] = t * mul; kb[1] = mul; kb[2] = t * mul;
    }
    for (int a = 0; a < 3; a++)
        for (int b = 0; b < 3; b++) p.w2d[a * 3 + b] = (float)(kb[a] * kb[b]);
    p.thr = (float)c->modulation_threshold;
    p.avg3 = c->avg_three_phase ? 1 : 0;
    if (c->encoding == ZIM_ENC_HETERODYNE3) {
        p.f0 = (int)c->freq[0]; p.f1 = (int)c->freq[1]; p.f2 = (int)c->freq[2];
        p.f12 = std::abs(p.f0 - p.f1); p.f23 = std::abs(p.f1 - p.f2);
        p.f1_gt_f2 = c->freq[1] > c->freq[2];
        p.f0_f12 = (float)((double)p.f0 / p.f12);
        p.f1_f23 = (float)((double)p.f1 / p.f23);
        p.f2_f23 = (float)((double)p.f2 / p.f23);
        p.inv_f12 = (float)(1.0 / p.f12);
        p.inv_f23 = (float)(1.0 / p.f23);
        p.inv_f1 = (float)(1.0 / p.f1);
        p.inv_f2 = (float)(1.0 / p.f2);
    } else if (c->encoding == ZIM_ENC_HIERARCHICAL) {
        for (int i = 1; i < c->n_freq; i++) {
            p.iratio[i] = (int)(c->freq[i] / c->freq[i - 1]);
            p.fratio[i] = (float)p.iratio[i];
        }
    } else {
        p.gray_bits = c->gray_bits;
        p.gray_base = c->shift_num[0];
        p.complementary = c->encoding == ZIM_ENC_GRAYCODE_COMPLEMENTARY;
    }
    p.hdr = c->enable_hdr ? 1 : 0;
    p.hdr_sat = (float)c->hdr_saturation_gray;
    p.hdr_min_amp = (float)c->hdr_min_amplitude;
}

// Four-quadrant arctangent of the wrapped phase.  The octant ratio
// t = min(|y|, |x|) / max(|y|, |x|) in [0, 1] gives atan(t) = t P(t^2) with P of
// degree 7, fitted for this kernel by iteratively reweighted least squares on
// Chebyshev nodes (absolute error 3.7e-8 in exact arithmetic, 1.4e-7 evaluated
// by FP32 Horner FMAs); the octant and quadrant follow by symmetry, with atan2's
// signed zeros (the sign bits of y and x) and 0 for (0, 0).  __fdividef is
// exact to 2 ulp for the divisor range of these sums (far below 2^126).
__device__ __forceinline__ float phase_atan2(float y, float x) {
    const float ax = fabsf(x), ay = fabsf(y);
    const float hi = fmaxf(ax, ay), lo = fminf(ax, ay);
    const float t = hi > 0.f ? __fdividef(lo, hi) : 0.f;
    const float s = t * t;
    float p = -0.004054566845297813f;
    p = fmaf(p, s, 0.021862957626581192f);
    p = fmaf(p, s, -0.0559123270213604f);
    p = fmaf(p, s, 0.0964219719171524f);
    p = fmaf(p, s, -0.1390862911939621f);
    p = fmaf(p, s, 0.19946566224098206f);
    p = fmaf(p, s, -0.33329859375953674f);
    p = fmaf(p, s, 0.9999993443489075f);
    float r = t * p;
    if (ay > ax) r = 0.5f * ZIM_PI_F - r;
    if (signbit(x)) r = ZIM_PI_F - r;
    return copysignf(r, y);
}

// --------------------------------------------------------------- rectify ----

// Decoded phase at source pixel o in exact integer + FP32 form: phase = 2 pi K16 / 16 +
// R.  post_smooth 0: as decoded; 3: the same for HDR decodes, whose invalid pixels
// (order -1) have phase 0.
__device__ __forceinline__ void decoded_tap(const int32_t* __restrict__ order, const float* __restrict__ res, size_t o,
                                            int post_smooth, int& K16, float& R) {
    const int k = __ldg(order + o);
    const bool zero = post_smooth == 3 && k < 0;
    K16 = zero ? 0 : 16 * k;
    R = zero ? 0.f : __ldg(res + o);
}

// setData remap of one rectified pixel without post-smooth: INTER_LINEAR of the
// phase with OpenCV's 1/32-pixel quantised weights and BORDER_CONSTANT 0,
// INTER_NEAREST of the order.  The phase is kept as an integer cycle count
// (exact: every weight is a multiple of 1/16384) plus an FP32 residual.
__device__ __forceinline__ void rectify_pixel(const int32_t* __restrict__ order, const float* __restrict__ res,
                                              int srows, int scols, float mx, float my, int post_smooth,
                                              int32_t& rbase, float& rres, int32_t& rorder) {
    int nx = __float2int_rn(mx), ny = __float2int_rn(my);
    int ko = 0;
    if (nx >= 0 && ny >= 0 && nx < scols && ny < srows) ko = __ldg(order + (size_t)ny * scols + nx);
    int sx = __float2int_rn(mx * 32.0f), sy = __float2int_rn(my * 32.0f);
    int x0 = sx >> 5, y0 = sy >> 5;
    int fx = sx & 31, fy = sy & 31;
    long long I = 0;
    float Rs = 0.f;
#pragma unroll
    for (int t = 0; t < 4; t++) {
        int xx = x0 + (t & 1), yy = y0 + (t >> 1);
        if (xx < 0 || yy < 0 || xx >= scols || yy >= srows) continue;
        int wq = ((t >> 1) ? fy : 32 - fy) * ((t & 1) ? fx : 32 - fx);
        if (wq == 0) continue;
        int K16;
        float R;
        decoded_tap(order, res, (size_t)yy * scols + xx, post_smooth, K16, R);
        I += (long long)wq * K16;
        Rs = fmaf((float)wq * (1.0f / 1024.0f), R, Rs);
    }
    // phase = 2*pi*I/16384 + Rs; split I = 16384*base + frac, frac in [-8192, 8192)
    long long base = (I + 8192) >> 14;  // floor((I + 8192) / 16384)
    int frac = (int)(I - (base << 14));
    rbase = (int32_t)base;
    rres = fmaf((float)frac, ZIM_TWO_PI_F / 16384.0f, Rs);
    rorder = ko;
}

// Post-smooth of the decoded phase once per source pixel, so that a rectified
// pixel reads 4 taps instead of 4 x 9: a tap is (K16, bits of R) with smoothed
// phase = 2 pi K16 / 16 + R, K16 = sum (1 2 1)x(1 2 1) * order (BORDER_REPLICATE), the
// two words together so that a tap is one load.
//
// HDR (JSLAB_PhaseShiftDecoder_V2.cpp:280-291): the blurred phase divided by the
// blurred validity (invalid pixels, order < 0, count as phase 0 with weight 0), 0
// at invalid pixels.  With W = sum of the valid [1 2 1]^2 weights and Kw = sum w
// k: phase = 2 pi Kw / W + 16 (sum w r / 16) / W, and Kw / W splits exactly into
// an integer q and remainder, so the tap keeps its form: K16 = 16 q, R = (2 pi
// rem + 16 Rw) / W.
//
// One warp per strip of SMOOTH_STRIP columns marching down rows [y0, y1): each
// row's values are loaded once, exchanged with the neighbour lanes by shuffles
// and added to the three rows they blur into.  30 -> 21 us at 2448x2048 (the HDR
// form 60 -> 25) against nine gathers per pixel; bound by load latency.
constexpr int SMOOTH_STRIP = 30;
template <bool HDR>
__device__ __forceinline__ void smooth_strip(const int32_t* __restrict__ order, const float* __restrict__ res, int rows,
                                             int cols, int strip, int y0, int y1, int2* __restrict__ taps) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int x = strip * SMOOTH_STRIP - 1 + lane, xc = min(max(x, 0), cols - 1);
    const bool writes = lane > 0 && lane < 31 && x < cols;
    auto off = [&](int y) { return (size_t)min(max(y, 0), rows - 1) * cols + xc; };
    int kn = __ldg(order + off(y0 - 1)), kc = 0;  // next row's order; the current one's (of the row to write)
    float rn = __ldg(res + off(y0 - 1));
    int A = 0, B = 0, WA = 0, WB = 0;  // integer sums under way (the row above, this row)
    float RA = 0.f, RB = 0.f;
    for (int y = y0 - 1; y <= y1; y++) {
        int k = kn;
        float r = rn;
        const int above = kc;
        kc = k;
        if (y < y1) {
            kn = __ldg(order + off(y + 1));
            rn = __ldg(res + off(y + 1));
        }
        int w = 1;
        if (HDR && k < 0) {
            k = w = 0;
            r = 0.f;
        }
        const int kh = __shfl_up_sync(full, k, 1) + 2 * k + __shfl_down_sync(full, k, 1);
        const float rl = __shfl_up_sync(full, r, 1), rr = __shfl_down_sync(full, r, 1);
        // taps in row-major order from zero, as nine sequential FMAs per output
        const float RF = fmaf(0.0625f, rr, fmaf(0.125f, r, fmaf(0.0625f, rl, RA)));
        RA = fmaf(0.125f, rr, fmaf(0.25f, r, fmaf(0.125f, rl, RB)));
        RB = fmaf(0.0625f, rr, fmaf(0.125f, r, fmaf(0.0625f, rl, 0.f)));
        const int F = A + kh;
        A = B + 2 * kh;
        B = kh;
        int WF = 16;
        if (HDR) {
            const int wh = __shfl_up_sync(full, w, 1) + 2 * w + __shfl_down_sync(full, w, 1);
            WF = WA + wh;
            WA = WB + 2 * wh;
            WB = wh;
        }
        if (y <= y0 || !writes) continue;
        int K16 = F;
        float R = RF;
        if (HDR) {
            if (above < 0) {
                K16 = 0;
                R = 0.f;
            } else {
                int q = F / WF;  // WF in [4, 16]
                int rem = F - q * WF;
                if (rem < 0) {
                    q--;
                    rem += WF;
                }
                K16 = 16 * q;
                R = fmaf((float)rem, ZIM_TWO_PI_F, 16.0f * RF) / (float)WF;
            }
        }
        taps[(size_t)(y - 1) * cols + x] = make_int2(K16, __float_as_int(R));
    }
}

// setData remap of one rectified pixel (see rectify_pixel) from smoothed taps.
// Bound by the latency of the gathers behind the map (a warp-uniform path without
// the border tests and conversions issued less and took the same time).
__device__ __forceinline__ void rectify_pixel_smoothed(const int2* __restrict__ taps, const int32_t* __restrict__ order,
                                                       int srows, int scols, float mx, float my, int32_t& rbase,
                                                       float& rres, int32_t& rorder) {
    const int nx = __float2int_rn(mx), ny = __float2int_rn(my);
    rorder = 0;
    if ((unsigned)nx < (unsigned)scols && (unsigned)ny < (unsigned)srows) rorder = __ldg(order + (size_t)ny * scols + nx);
    const int sx = __float2int_rn(mx * 32.0f), sy = __float2int_rn(my * 32.0f);
    const int x0 = sx >> 5, y0 = sy >> 5, fx = sx & 31, fy = sy & 31;
    // a tap of weight 0 or outside the image is not read
    const bool xl = (unsigned)x0 < (unsigned)scols, xr = fx && (unsigned)(x0 + 1) < (unsigned)scols;
    const bool yt = (unsigned)y0 < (unsigned)srows, yb = fy && (unsigned)(y0 + 1) < (unsigned)srows;
    const int2* q = taps + (ptrdiff_t)y0 * scols + x0;
    const int2 z = make_int2(0, 0);
    const int2 t00 = yt && xl ? __ldg(q) : z, t01 = yt && xr ? __ldg(q + 1) : z;
    const int2 t10 = yb && xl ? __ldg(q + scols) : z, t11 = yb && xr ? __ldg(q + scols + 1) : z;
    const int w11 = fy * fx, w10 = 32 * fy - w11, w01 = 32 * fx - w11, w00 = 1024 - 32 * fy - w01;
    // phase = 2*pi*I/16384 + Rs; split I = 16384*base + frac, frac in [-8192, 8192)
    const long long I = (long long)w00 * t00.x + (long long)w01 * t01.x + (long long)w10 * t10.x +
                        (long long)w11 * t11.x + 8192;
    float Rs = fmaf((float)w00 * (1.0f / 1024.0f), __int_as_float(t00.y), 0.f);
    Rs = fmaf((float)w01 * (1.0f / 1024.0f), __int_as_float(t01.y), Rs);
    Rs = fmaf((float)w10 * (1.0f / 1024.0f), __int_as_float(t10.y), Rs);
    Rs = fmaf((float)w11 * (1.0f / 1024.0f), __int_as_float(t11.y), Rs);
    const int frac = ((int)I & 16383) - 8192;
    rbase = (int32_t)(I >> 14);
    rres = fmaf((float)frac, ZIM_TWO_PI_F / 16384.0f, Rs);
}

// ----------------------------------------------------------------- match ----

__device__ __forceinline__ float phase_diff(int bR, float rR, int bL, float rL) {
    // (2 pi bR + rR) - (2 pi bL + rL) with the integer cycles subtracted exactly
    return fmaf((float)(bR - bL), ZIM_TWO_PI_F, rR - rL);
}

// Monotone spans.  Within a right row the rectified phase of one fringe order
// normally rises column by column.  When the order's span [lo, hi] holds only
// pixels of that order and every step to the next column rises by more than
// MATCH_MONO_MARGIN (verified per row and order by match_spans_check), the
// float differences d(c) = phase_R(c) - phase_L computed by phase_diff are
// strictly increasing in c for any left pixel whose phase lies within 1024
// cycles of the span (the rounding of each d is below half the margin), so
// |d| falls, then rises, and its first minimum is at the sign change of d: a
// bracketing search finds the same column as the reference's scan over every
// candidate (ties keep the earlier column, as the scan's strict < does).
// Spans that fail the check are scanned in full.
constexpr float MATCH_MONO_MARGIN = 2e-3f;

// One left pixel against a right row staged in shared memory (s_ord, s_ph =
// (base, bits of the residual); cols columns) with the per-order column spans [s_lo, s_hi] and the
// spans' failed-check flags s_bad (null: always the full scan): the first
// column of minimum |phase_R - phase_L| among right pixels of the same order
// (strict <), rejected if min >= grad_threshold or the column is < 2 or
// >= cols - 1, then the reference's three-point sub-pixel refinement.
// dx_off is (left window x) - (right window x) for the ROI path
// (startCalculate_v2_roi, V2.cpp:719-778: global left x - global right x - delta).
__device__ __forceinline__ void match_pixel(int j, int k, int bL, float rL, const int* s_ord, const int2* s_ph,
                                            const int* s_lo, const int* s_hi, const int* s_bad,
                                            int cols, int pha_f, float grad_threshold, float& d, int& best,
                                            int dx_off = 0) {
    d = 0.f;
    best = -1;
    if (k < 1 || k > pha_f) return;
    auto diff = [&](int c) {
        const int2 q = s_ph[c];
        return phase_diff(q.x, __int_as_float(q.y), bL, rL);
    };
    const int lo = s_lo[k], hi = s_hi[k];
    if (lo > hi) return;
    float min_cost = 1e9f, c0 = 0.f, c1 = 0.f, c2 = 0.f;
    int bj = -1, miss = 0;  // miss: the costs beside bj still to evaluate (1 left, 2 right)
    if (s_bad && !s_bad[k] && abs(s_ph[lo].x - bL) < 1024 && abs(s_ph[hi].x - bL) < 1024) {
        // d rises strictly: the sign change between adjacent columns a and b.  The
        // phase is close to linear over a span, so the first probe interpolates
        // and the next two try the neighbour; from the fourth on the bracket halves.
        int a = lo, b = hi;
        float da = diff(a), db = diff(b);
        if (!(da < 0.f) || db < 0.f) {
            bj = da < 0.f ? hi : lo;
            c1 = da < 0.f ? db : da;
            miss = 3;
        } else {
            int m = a + (int)(__fdividef(da, da - db) * (float)(b - a));
            for (int step = 0; b - a > 1; step++) {
                m = step < 3 ? min(max(m, a + 1), b - 1) : (a + b) >> 1;
                const float dm = diff(m);
                if (dm < 0.f) {
                    a = m++;
                    da = dm;
                } else {
                    b = m--;
                    db = dm;
                }
            }
            const bool right = fabsf(db) < fabsf(da);  // a tie keeps the earlier column
            bj = right ? b : a;
            c1 = right ? db : da;
            c0 = da;  // of the left neighbour when bj = b
            c2 = db;  // of the right neighbour when bj = a
            miss = right ? 2 : 1;
        }
        min_cost = fabsf(c1);
    } else {
        for (int c = lo; c <= hi; c++) {
            if (s_ord[c] != k) continue;
            const float cost = fabsf(diff(c));
            if (cost < min_cost) {
                min_cost = cost;
                bj = c;
            }
        }
        miss = 3;
        if (bj >= 0) c1 = diff(bj);
    }
    if (bj >= 0 && min_cost < grad_threshold && bj >= 2 && bj < cols - 1) {
        if (miss & 1) c0 = diff(bj - 1);
        if (miss & 2) c2 = diff(bj + 1);
        float num = c1 * (c0 - c2);
        float den = 2.0f * (c0 - c1) * (c1 - c2);
        float delta = fabsf(den) > 1e-9f ? num / den : 0.f;
        d = (float)(j - bj + dx_off) - delta;
        best = bj;
    }
}

// Per-order column spans of a staged right row (shared atomics).  Callers
// initialise s_lo = INT_MAX, s_hi = -1, s_bad = 0 and sync before, and sync
// after, then run match_spans_check (and sync again).  A span's first column
// is the first column of one of its order's runs and its last the last of
// one, so only run starts update s_lo and only run ends s_hi: about two
// atomics per run instead of one per pixel (a warp's lanes nearly always
// share an order, and same-address atomics serialise).
__device__ __forceinline__ void match_spans(const int* s_ord, int cols, int pha_f, int* s_lo, int* s_hi, int tid,
                                            int nthreads) {
    for (int j = tid; j < cols; j += nthreads) {
        int k = s_ord[j];
        if (k >= 0 && k <= pha_f) {
            if (j == 0 || s_ord[j - 1] != k) atomicMin(&s_lo[k], j);
            if (j == cols - 1 || s_ord[j + 1] != k) atomicMax(&s_hi[k], j);
        }
    }
}

// Marks in s_bad every order whose span holds a pixel of another order or a
// step that does not rise by MATCH_MONO_MARGIN (see match_pixel).  A foreign
// run inside a span always follows a pixel of the span's order, so checking
// each pixel against its right neighbour finds it.
__device__ __forceinline__ void match_spans_check(const int* s_ord, const int2* s_ph, int cols, int pha_f, const int* s_hi,
                                                  int* s_bad, int tid, int nthreads) {
    for (int j = tid; j + 1 < cols; j += nthreads) {
        const int k = s_ord[j];
        if (k < 0 || k > pha_f || j >= s_hi[k]) continue;
        const int2 a = s_ph[j], b = s_ph[j + 1];
        if (s_ord[j + 1] != k || !(phase_diff(b.x, __int_as_float(b.y), a.x, __int_as_float(a.y)) > MATCH_MONO_MARGIN))
            s_bad[k] = 1;
    }
}

// -------------------------------------------------------- pixel rays ----
// An organised cloud from one camera: cloud pixel (u, v) looks from the origin
// along R (u + ox - cx, v + oy - cy, f).  A point p seen along the ray of
// pixel b and a query q near the ray of pixel a satisfy
// |p - q| >= |q| sin(angle(a, b)) - dev(q) - dev(p) (dev: distance from the own
// ray), and with |a x b| >= f |b - a|, |b| <= |a| + |b - a|:
// sin(angle) >= f |b - a| / (|a| (|a| + |b - a|)), increasing in |b - a|.
// The window paths of the filters use this to stop scanning a pixel window.

struct RayParams {
    float cx, cy, f, R[9];
    int ox, oy;
};

__device__ __forceinline__ void ray_dir(const RayParams& r, int u, int v, float& ax, float& ay, float& az) {
    const float x = (float)(u + r.ox) - r.cx, y = (float)(v + r.oy) - r.cy;
    ax = fmaf(r.R[0], x, fmaf(r.R[1], y, r.R[2] * r.f));
    ay = fmaf(r.R[3], x, fmaf(r.R[4], y, r.R[5] * r.f));
    az = fmaf(r.R[6], x, fmaf(r.R[7], y, r.R[8] * r.f));
}

// Distance of p from the line through the origin along a: |p x a| / |a|.
__device__ __forceinline__ float ray_dev(float px, float py, float pz, float ax, float ay, float az) {
    const float cx = fmaf(py, az, -pz * ay), cy = fmaf(pz, ax, -px * az), cz = fmaf(px, ay, -py * ax);
    return sqrtf(fmaf(cx, cx, fmaf(cy, cy, cz * cz))) * rsqrtf(fmaf(ax, ax, fmaf(ay, ay, az * az)));
}

inline RayParams ray_params(const zim_ray_model& r) {
    RayParams p;
    p.cx = r.cx; p.cy = r.cy; p.f = r.f;
    for (int a = 0; a < 9; a++) p.R[a] = r.R[a];
    p.ox = r.ox; p.oy = r.oy;
    return p;
}

// half-size and offset count of the window-pass windows (the offsets
// themselves, ordered by length, then row, then column, are a compile-time
// table beside the kernels)
constexpr int SPIRAL_R = 7;
constexpr int SPIRAL_N = (2 * SPIRAL_R + 1) * (2 * SPIRAL_R + 1) - 1;

// -------------------------------------------------- median + reprojection ----

constexpr int RX = 32, RY = 8;  // pixel-filter tile

struct ReprojParams {
    float q03, q13, q23, q32, q33;
    double dq03, dq13, dq23, dq32, dq33;
    float r1[9];
    float min_depth, max_depth;
    double dmin_depth, dmax_depth;
    int use_rectified, use_median;
    int model;                 // 0: Q matrix; 1: per-pixel polynomial maps
    double dr1[9];
    const float4* poly[3];     // x, y, z coefficient maps (c0, c1, c2, c3) per rectified pixel
    // ROI tiles (startCalculate_v2_roi): the disparity tile starts at rectified
    // pixel (ox, oy); points are made only where roi_mask (rectified frame,
    // gstride pixels per row) is non-zero.  Whole frames: 0, 0, null.
    int ox, oy, gstride;
    const uint8_t* roi_mask;
};

inline void reproj_params(const double Q[16], const double R1[9], const zim_recon_config* cfg, ReprojParams& p) {
    p.q03 = (float)Q[3]; p.q13 = (float)Q[7]; p.q23 = (float)Q[11];
    p.q32 = (float)Q[14]; p.q33 = (float)Q[15];
    p.dq03 = Q[3]; p.dq13 = Q[7]; p.dq23 = Q[11]; p.dq32 = Q[14]; p.dq33 = Q[15];
    for (int i = 0; i < 9; i++) p.r1[i] = (float)R1[i];
    p.min_depth = (float)cfg->min_depth;
    p.max_depth = (float)cfg->max_depth;
    p.dmin_depth = cfg->min_depth;
    p.dmax_depth = cfg->max_depth;
    p.use_rectified = cfg->use_rectified_coords != 0;
    p.use_median = cfg->use_disp_median_filter != 0;
    p.model = cfg->reproject_model;
    for (int i = 0; i < 9; i++) p.dr1[i] = R1[i];
    p.poly[0] = p.poly[1] = p.poly[2] = nullptr;
    p.ox = p.oy = p.gstride = 0;
    p.roi_mask = nullptr;
}

// Per-pixel polynomial calibration, evaluateV2CalibPoint
// (JSLAB_PhaseEpipolarReconstructor_V2.cpp:13-76): the coefficient maps carry
// a model tag in c3 of the x map (-1 inverse depth, -2 fitted ray, -3 z-linear
// x/y) and of the z map (-1 inverse depth, -4 rational depth); untagged maps
// are cubics in d.  Evaluated in FP64 in the reference's operation order with
// every product and sum rounded separately (no contraction), so the result is
// the same bit pattern as a strict IEEE evaluation on the host.
__device__ __forceinline__ double pm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double pa(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ bool poly_tag(float c, float tag) { return fabsf(c - tag) < 1e-6f; }

__device__ __forceinline__ bool poly_point(const float4& cx, const float4& cy, const float4& cz, double d, double& X,
                                           double& Y, double& Z) {
    if (fabsf(cz.x) <= 1e-9 && fabsf(cz.y) <= 1e-9 && fabsf(cz.z) <= 1e-9 && fabsf(cz.w) <= 1e-9) return false;
    const double z0 = cz.x, z1 = cz.y, z2 = cz.z, z3 = cz.w;
    if (poly_tag(cx.w, -1.0f) || poly_tag(cx.w, -2.0f)) {
        const double d2 = pm(d, d);
        if (poly_tag(cx.w, -1.0f) || poly_tag(cz.w, -1.0f)) {
            // inverse depth: cubic (x-map tag -1) or quadratic (x-map tag -2, z-map tag -1)
            double iz = pa(pa(z0, pm(z1, d)), pm(z2, d2));
            if (poly_tag(cx.w, -1.0f)) iz = pa(iz, pm(pm(z3, d2), d));
            if (!isfinite(iz) || fabs(iz) < 1e-12) return false;
            Z = 1.0 / iz;
        } else {
            Z = pa(pa(pa(z0, pm(z1, d)), pm(z2, d2)), pm(pm(z3, d2), d));
        }
        X = pm((double)cx.x, Z);
        Y = pm((double)cy.x, Z);
    } else if (poly_tag(cx.w, -3.0f)) {
        if (poly_tag(cz.w, -4.0f)) {
            const double den = pa(pm(z1, d), 1.0);
            if (!isfinite(den) || fabs(den) < 1e-12) return false;
            Z = z0 / den;
        } else {
            const double d2 = pm(d, d), d3 = pm(d2, d);
            Z = pa(pa(pa(z0, pm(z1, d)), pm(z2, d2)), pm(z3, d3));
        }
        X = pa(pm((double)cx.x, Z), (double)cx.y);
        Y = pa(pm((double)cy.x, Z), (double)cy.y);
    } else if (poly_tag(cz.w, -1.0f)) {
        const double iz = pa(pa(z0, pm(z1, d)), pm(pm(z2, d), d));
        if (!isfinite(iz) || fabs(iz) < 1e-12) return false;
        Z = 1.0 / iz;
        X = pm((double)cx.x, Z);
        Y = pm((double)cy.x, Z);
    } else {
        const double d2 = pm(d, d), d3 = pm(d2, d);
        X = pa(pa(pa((double)cx.x, pm((double)cx.y, d)), pm((double)cx.z, d2)), pm((double)cx.w, d3));
        Y = pa(pa(pa((double)cy.x, pm((double)cy.y, d)), pm((double)cy.z, d2)), pm((double)cy.w, d3));
        Z = pa(pa(pa(z0, pm(z1, d)), pm(z2, d2)), pm(z3, d3));
    }
    return isfinite(X) && isfinite(Y) && isfinite(Z);
}

// startCalculate_v2's per-pixel body (:505-547): polynomial point, optional
// R1^T rotation, depth gate on the reported z.
__device__ __forceinline__ void poly_reproject_point(const ReprojParams& p, size_t o, float d, float& ox, float& oy,
                                                     float& oz, uint8_t& m) {
    const float4 cz = __ldg(p.poly[2] + o);
    double X, Y, Z;
    if (!poly_point(__ldg(p.poly[0] + o), __ldg(p.poly[1] + o), cz, (double)d, X, Y, Z)) return;
    if (p.use_rectified) {
        if (Z > p.dmin_depth && Z < p.dmax_depth) { ox = (float)X; oy = (float)Y; oz = (float)Z; m = 1; }
        return;
    }
    const double rx = pa(pa(pm(p.dr1[0], X), pm(p.dr1[3], Y)), pm(p.dr1[6], Z));
    const double ry = pa(pa(pm(p.dr1[1], X), pm(p.dr1[4], Y)), pm(p.dr1[7], Z));
    const double rz = pa(pa(pm(p.dr1[2], X), pm(p.dr1[5], Y)), pm(p.dr1[8], Z));
    if (rz > p.dmin_depth && rz < p.dmax_depth) { ox = (float)rx; oy = (float)ry; oz = (float)rz; m = 1; }
}

__device__ __forceinline__ void cswap(float& a, float& b) {
    float lo = fminf(a, b), hi = fmaxf(a, b);
    a = lo;
    b = hi;
}

// Sorts five values (nine exchanges).
__device__ __forceinline__ void sort5(float (&v)[5]) {
    cswap(v[0], v[3]); cswap(v[1], v[4]); cswap(v[0], v[2]); cswap(v[1], v[3]); cswap(v[0], v[1]);
    cswap(v[2], v[4]); cswap(v[1], v[2]); cswap(v[3], v[4]); cswap(v[2], v[3]);
}

// Odd-even merges (Batcher) of two sorted lists of two, three and five values.
__device__ __forceinline__ void merge2(float a0, float a1, float b0, float b1, float (&o)[4]) {
    cswap(a0, b0);
    cswap(a1, b1);
    cswap(a1, b0);
    o[0] = a0; o[1] = a1; o[2] = b0; o[3] = b1;
}
__device__ __forceinline__ void merge3(float a0, float a1, float a2, float b0, float b1, float b2, float (&o)[6]) {
    float d[4];
    merge2(a0, a2, b0, b2, d);
    cswap(a1, b1);
    cswap(a1, d[1]);
    cswap(b1, d[2]);
    o[0] = d[0]; o[1] = a1; o[2] = d[1]; o[3] = b1; o[4] = d[2]; o[5] = d[3];
}
__device__ __forceinline__ void merge5(const float (&a)[5], const float (&b)[5], float (&o)[10]) {
    float d[6], e[4];
    merge3(a[0], a[2], a[4], b[0], b[2], b[4], d);
    merge2(a[1], a[3], b[1], b[3], e);
    o[0] = d[0];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        o[2 * k + 1] = fminf(e[k], d[k + 1]);
        o[2 * k + 2] = fmaxf(e[k], d[k + 1]);
    }
    o[9] = d[5];
}

// Two horizontally adjacent 5x5 windows share 20 values.  A shared value of
// rank r among those 20 has rank r .. r + 5 in either window, so only ranks
// 8..13 can be a window's median (rank 13 of 25); with the 7 lower shared
// values below them and at most 5 own values among the rest, each window's
// median is the median (rank 6) of those 6 and its own 5-value column.
// mid6: ranks 8..13, in order, of two sorted lists of ten.  The first step of a
// bitonic merge splits the 20 into the lower and the upper ten, a second one each
// into halves; the upper five of the lower ten and the lower five of the upper
// ten hold them (exchanges whose results are not used cost nothing).
__device__ __forceinline__ void mid6(const float (&a)[10], const float (&b)[10], float (&m)[6]) {
    float lo[5], hi[5];
#pragma unroll
    for (int i = 0; i < 5; i++) {
        lo[i] = fmaxf(fminf(a[i], b[9 - i]), fminf(a[i + 5], b[4 - i]));
        hi[i] = fminf(fmaxf(a[i], b[9 - i]), fmaxf(a[i + 5], b[4 - i]));
    }
    sort5(lo);
    sort5(hi);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        m[i] = lo[2 + i];
        m[3 + i] = hi[i];
    }
}

// Median (rank 6) of a sorted list of six and a sorted list of five.
__device__ __forceinline__ float median_6_5(const float (&m)[6], const float (&o)[5]) {
    float r = m[5];
#pragma unroll
    for (int i = 0; i < 5; i++) r = fminf(r, fmaxf(m[i], o[4 - i]));
    return r;
}

// Q (or polynomial-map) reprojection of one pixel's disparity; (gx, gy) its
// rectified-frame pixel, go its index in the maps.
__device__ __forceinline__ void reproject_pixel(const ReprojParams& p, int gx, int gy, size_t go, float d, float& ox,
                                                float& oy, float& oz, uint8_t& m) {
    ox = oy = oz = 0.f;
    m = 0;
    // the reference gates |d| < 1e-5 on the disparity widened to double: the
    // float 1e-5 lies below that bound and the next float above it, so > decides
    // the same (a conversion to FP64 per pixel held the kernel at the FP64 pipe)
    const bool has_d = fabsf(d) > 1e-5f && (!p.roi_mask || p.roi_mask[go]);
    if (p.model == 1) {
        if (has_d) poly_reproject_point(p, go, d, ox, oy, oz, m);
    } else if (has_d) {
        float X, Y, Z;
        float w = fmaf(p.q32, d, p.q33);
        if (fabsf(w) < 1e-2f * (fabsf(p.q32 * d) + fabsf(p.q33))) {
            // near-zero disparity denominator: FP64 divide
            double wd = fma(p.dq32, (double)d, p.dq33);
            double iw = 1.0 / wd;
            X = (float)(((double)gx + p.dq03) * iw);
            Y = (float)(((double)gy + p.dq13) * iw);
            Z = (float)(p.dq23 * iw);
            double zz = p.dq23 * iw;
            if (p.use_rectified) {
                if (zz > p.dmin_depth && zz < p.dmax_depth) { ox = X; oy = Y; oz = Z; m = 1; }
            } else {
                double xx = ((double)gx + p.dq03) * iw, yy = ((double)gy + p.dq13) * iw;
                double rx = fma((double)p.r1[0], xx, fma((double)p.r1[3], yy, (double)p.r1[6] * zz));
                double ry = fma((double)p.r1[1], xx, fma((double)p.r1[4], yy, (double)p.r1[7] * zz));
                double rz = fma((double)p.r1[2], xx, fma((double)p.r1[5], yy, (double)p.r1[8] * zz));
                if (rz > p.dmin_depth && rz < p.dmax_depth) { ox = (float)rx; oy = (float)ry; oz = (float)rz; m = 1; }
            }
        } else {
            float iw = 1.0f / w;
            X = ((float)gx + p.q03) * iw;
            Y = ((float)gy + p.q13) * iw;
            Z = p.q23 * iw;
            if (p.use_rectified) {
                if (Z > p.min_depth && Z < p.max_depth) { ox = X; oy = Y; oz = Z; m = 1; }
            } else {
                float rx = fmaf(p.r1[0], X, fmaf(p.r1[3], Y, p.r1[6] * Z));
                float ry = fmaf(p.r1[1], X, fmaf(p.r1[4], Y, p.r1[7] * Z));
                float rz = fmaf(p.r1[2], X, fmaf(p.r1[5], Y, p.r1[8] * Z));
                if (rz > p.min_depth && rz < p.max_depth) { ox = rx; oy = ry; oz = rz; m = 1; }
            }
        }
    }
}

// 5x5 median (replicate border) + Q reprojection, one warp per strip of
// MSTRIP columns marching down rows [y0, y1).  Lane t holds columns 2t and 2t + 1
// of the strip's 64 (the strip and three on either side): their five rows are
// sorted and merged once per row, and the neighbours' sorted columns come by
// shuffles, so a row costs each lane two five-value sorts, a merge and half of the
// selections of its two output pixels (2t + 1, 2t + 2).  The points leave through
// the warp's shared buffer, so the stores are contiguous.
//
// Bound by the compare instructions (the ALU pipe): about 70 per pixel, against
// 203 of a selection by elimination per pixel pair without shared sorts.
// Before / now, median and reprojection: 99 / 50 us at 2501x2092 pixels, 244 / 112
// at 4185x3064 (three CTAs per SM; 57 and 124 us with the registers for two).
constexpr int MSTRIP = 58;
constexpr int MED_WARPS = 8;
struct MedianSmem {
    float xyz[MED_WARPS][3 * MSTRIP];
    float d[MED_WARPS][MSTRIP];
    uint8_t m[MED_WARPS][64];
};

__device__ __forceinline__ void median_reproject_strip(const float* __restrict__ disp, int rows, int cols,
                                                       const ReprojParams& p, int strip, int y0, int y1, int warp,
                                                       MedianSmem& sm, float* __restrict__ disp_out,
                                                       float* __restrict__ xyz, uint8_t* __restrict__ mask) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int first = MSTRIP * strip, n = min(MSTRIP, cols - first);  // the strip's columns
    const int ca = min(max(first - 3 + 2 * lane, 0), cols - 1), cb = min(max(first - 2 + 2 * lane, 0), cols - 1);
    float* sx = sm.xyz[warp];
    float* sd = sm.d[warp];
    uint8_t* smk = sm.m[warp];
    auto load = [&](int y, float& a, float& b) {
        const float* r = disp + (size_t)min(max(y, 0), rows - 1) * cols;
        a = __ldg(r + ca);
        b = __ldg(r + cb);
    };
    float a[5], b[5], na, nb;
#pragma unroll
    for (int r = 0; r < 4; r++) load(y0 - 2 + r, a[r + 1], b[r + 1]);
    load(y0 + 2, na, nb);
    const int k0 = 2 * lane - 2;  // first output pixel in the strip: column 2t + 1 less the three
    for (int y = y0; y < y1; y++) {
#pragma unroll
        for (int r = 0; r < 4; r++) {
            a[r] = a[r + 1];
            b[r] = b[r + 1];
        }
        a[4] = na;
        b[4] = nb;
        if (y + 1 < y1) load(y + 3, na, nb);
        float d0, d1;
        if (p.use_median) {
            float s0[5], s1[5], own0[5], own1[5], P[10], Q[10], m[6];
#pragma unroll
            for (int r = 0; r < 5; r++) {
                s0[r] = a[r];
                s1[r] = b[r];
            }
            sort5(s0);
            sort5(s1);
            merge5(s0, s1, P);
#pragma unroll
            for (int r = 0; r < 10; r++) Q[r] = __shfl_down_sync(full, P[r], 1);
#pragma unroll
            for (int r = 0; r < 5; r++) {
                own0[r] = __shfl_up_sync(full, s1[r], 1);
                own1[r] = __shfl_down_sync(full, s0[r], 2);
            }
            mid6(P, Q, m);
            d0 = median_6_5(m, own0);
            d1 = median_6_5(m, own1);
        } else {
            d0 = b[2];
            d1 = __shfl_down_sync(full, a[2], 1);
        }
        __syncwarp();
#pragma unroll
        for (int l = 0; l < 2; l++) {
            const int k = k0 + l;
            if (k < 0 || k >= n) continue;
            const float d = l ? d1 : d0;
            // rectified-frame pixel (ROI tiles are offset) and its index in the maps
            const int gx = first + k + p.ox, gy = y + p.oy;
            const size_t go = p.gstride ? (size_t)gy * p.gstride + gx : (size_t)y * cols + first + k;
            float X, Y, Z;
            uint8_t v;
            reproject_pixel(p, gx, gy, go, d, X, Y, Z, v);
            sx[3 * k] = X;
            sx[3 * k + 1] = Y;
            sx[3 * k + 2] = Z;
            sd[k] = d;
            smk[k] = v;
        }
        __syncwarp();
        const size_t o = (size_t)y * cols + first;
#pragma unroll
        for (int u = 0; u < (3 * MSTRIP + 31) / 32; u++)
            if (lane + 32 * u < 3 * n) xyz[3 * o + lane + 32 * u] = sx[lane + 32 * u];
#pragma unroll
        for (int u = 0; u < 2; u++)
            if (lane + 32 * u < n) {
                if (disp_out) disp_out[o + lane + 32 * u] = sd[lane + 32 * u];
                mask[o + lane + 32 * u] = smk[lane + 32 * u];
            }
    }
}

// ------------------------------------------------- pixel-window filters ----

// getGaussianKernel(3, 0.7, CV_32F) outer-product weights: corner, edge, centre.
inline void px_gaussian_weights(float& w00, float& w01, float& w11) {
    double t = std::exp(-0.5 / (0.7 * 0.7));
    double mul = 1.0 / (2.0 * t + 1.0);
    float k0 = (float)(t * mul), k1 = (float)mul;
    w00 = k0 * k0;
    w01 = k0 * k1;
    w11 = k1 * k1;
}

// 3x3 point-cloud Gaussian (sigma 0.7 px): neighbour used if valid and
// |x_n - x_c| < 3; output sum(w p) / sum(w) if sum(w) > 0.8, else 0; borders 0.
// The weighted mean is accumulated as p_c + sum(w (p_n - p_c)) / sum(w), the same
// value with millimetre-scale FP32 sums.
//
// One warp per strip of PXG_STRIP columns marching down rows [y0, y1): a row's
// points are loaded once (invalid ones with x = NaN, which fails the test), the
// neighbours' come by shuffles, and three rows stay in registers: 132 -> 110 us at
// 4185x3064 against nine gathers per pixel.  Bound by instruction issue.
constexpr int PXG_STRIP = 30;
__device__ __forceinline__ void px_gaussian_strip(const float* __restrict__ xyz, const uint8_t* __restrict__ mask,
                                                  int rows, int cols, int strip, int y0, int y1, float w00, float w01,
                                                  float w11, float* __restrict__ out, uint8_t* __restrict__ mask_out) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int x = strip * PXG_STRIP - 1 + lane;
    const bool col = x >= 0 && x < cols, writes = lane > 0 && lane < 31 && x < cols;
    float nx = 0.f, ny = 0.f, nz = 0.f;
    bool nv = false;
    auto load = [&](int y) {
        nv = false;
        if (col && y >= 0 && y < rows) {
            const size_t o = (size_t)y * cols + x;
            nx = __ldg(xyz + 3 * o);
            ny = __ldg(xyz + 3 * o + 1);
            nz = __ldg(xyz + 3 * o + 2);
            nv = __ldg(mask + o) != 0;
        }
    };
    float p[3][3][3] = {};  // row above, centre row, row below; column; coordinate
    bool v1 = false, v2 = false;
    auto shift_in = [&]() {
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
            for (int b = 0; b < 3; b++)
#pragma unroll
                for (int c = 0; c < 3; c++) p[a][b][c] = p[a + 1][b][c];
        v1 = v2;
        v2 = nv;
        p[2][1][0] = nv ? nx : __int_as_float(0x7fc00000);
        p[2][1][1] = ny;
        p[2][1][2] = nz;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            p[2][0][c] = __shfl_up_sync(full, p[2][1][c], 1);
            p[2][2][c] = __shfl_down_sync(full, p[2][1][c], 1);
        }
    };
    load(y0 - 1);
    shift_in();
    load(y0);
    shift_in();
    load(y0 + 1);
    for (int y = y0; y < y1; y++) {
        shift_in();
        if (y + 1 < y1) load(y + 2);
        const float cx = p[1][1][0], cy = p[1][1][1], cz = p[1][1][2];
        float sx = 0.f, sy = 0.f, sz = 0.f, cnt = 0.f;
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) {
                const float dx = p[a][b][0] - cx;
                if (fabsf(dx) < 3.0f) {
                    const float w = (a == 1 && b == 1) ? w11 : ((a == 1 || b == 1) ? w01 : w00);
                    sx = fmaf(dx, w, sx);
                    sy = fmaf(p[a][b][1] - cy, w, sy);
                    sz = fmaf(p[a][b][2] - cz, w, sz);
                    cnt += w;
                }
            }
        if (!writes) continue;
        const bool keep = v1 && x >= 1 && y >= 1 && x < cols - 1 && y < rows - 1 && cnt > 0.8f;
        const size_t o = (size_t)y * cols + x;
        out[3 * o] = keep ? cx + sx / cnt : 0.f;
        out[3 * o + 1] = keep ? cy + sy / cnt : 0.f;
        out[3 * o + 2] = keep ? cz + sz / cnt : 0.f;
        if (mask_out) mask_out[o] = keep ? 1 : 0;
    }
}

// Radius outlier filter over a tile of RX columns and TH rows (a multiple of RY)
// from (x0, y0) with the RX * RY threads of a block: keep a valid point if at least
// min_nb valid neighbours (not itself) of its (2 hw + 1)^2 window lie within
// sqrt(r2).  The tile and its hw halo are staged in shared memory (ror_smem_bytes)
// as float4 with invalid and off-image pixels NaN, so a neighbour test is one
// shared load and an FP32 distance that compares false for NaN.  The point itself
// counts (distance 0), so the count including it must reach min_nb + 1 (with min_nb <= 0
// every valid point stays).  Ends past the last shared read.
//
// Bound by issue, staging first.  The default filter (11 x 11 window, 10 neighbours)
// at 4185x3064: 372 us with tiles of 8 rows scanned row by row, 302 with rings, 200
// with rings and tiles of 32 rows, 147 with the count checked every four neighbours
// and no division in the staging (every eight: 177).
//
// WIDE (half-windows above ROR_WIDE): ROR_RINGS rings, then the rest of the window row
// by row.  A long ring has four bases to step and its count to test every four
// neighbours; where nobody has enough, a window of 91 took 33.0 ms in rings at
// 2448x2048, 21.8 row by row and 21.5 so (41: 3.60, 3.49, 3.49), and where the first
// rings settle it all are the rings' (91, 5 mm: 1.57).  Narrow windows in rings alone:
// the second loop's registers cost the 11 x 11 filter 15 %.
constexpr int ROR_WIDE = 10, ROR_RINGS = 6;
// (The wide form also takes a radius whose square is infinite.)
inline bool ror_wide(int hw, float radius) { return hw > ROR_WIDE || !(radius * radius < INFINITY); }
__host__ __device__ inline size_t ror_smem_bytes(int hw, int th) {
    return (size_t)(RX + 2 * hw) * (th + 2 * hw) * sizeof(float4);
}

template <bool WIDE>
__device__ __forceinline__ void ror_tile(const float* __restrict__ xyz, const uint8_t* __restrict__ mask, int rows,
                                         int cols, int x0, int y0, int TH, int tid, float r2, int min_nb, int hw,
                                         float4* sp, float* __restrict__ out, uint8_t* __restrict__ mask_out) {
    const int TW = RX + 2 * hw;
    const int sy = RX * RY / TW, sx = RX * RY - sy * TW;  // a step of the block in rows and columns
    int gy = tid / TW, gx = tid - gy * TW + x0 - hw;
    gy += y0 - hw;
    for (int t = tid; t < TW * (TH + 2 * hw); t += RX * RY) {
        float4 v = make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
        if (gx >= 0 && gy >= 0 && gx < cols && gy < rows) {
            const size_t q = (size_t)gy * cols + gx;
            const float px = __ldg(xyz + 3 * q), py = __ldg(xyz + 3 * q + 1), pz = __ldg(xyz + 3 * q + 2);
            if (__ldg(mask + q)) v = make_float4(px, py, pz, 1.f);
        }
        sp[t] = v;
        gx += sx;
        gy += sy;
        if (gx >= x0 + RX + hw) {
            gx -= TW;
            gy++;
        }
    }
    __syncthreads();
    const int tx = tid % RX, x = x0 + tx;
    for (int ty = tid / RX; ty < TH; ty += RY) {
        const int y = y0 + ty;
        if (x >= cols || y >= rows) break;
        const float4* centre = sp + (ty + hw) * TW + tx + hw;
        const float4 c = *centre;
        bool keep = false;
        if (c.w != 0.f) {
            // rings of the window from the point outwards, until enough are near: on
            // a surface the nearest pixels settle it
            int cnt = 1;  // the point itself
            auto test = [&](const float4& p) {
                const float dx = c.x - p.x, dy = c.y - p.y, dz = c.z - p.z;
                cnt += fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= r2 ? 1 : 0;
            };
            if (WIDE && !(r2 < INFINITY)) {  // by its own distance, which is no number at infinity
                cnt = 0;
                test(c);
            }
            const int nr = WIDE ? min(hw, ROR_RINGS) : hw;
            for (int r = 1; r <= nr && cnt <= min_nb; r++) {
                const float4* a = centre - r * TW - r;  // the four sides, one step each
                const float4* b = centre + r * TW + r;
                const float4* l = centre + r * TW - r;
                const float4* g = centre - r * TW + r;
#pragma unroll 2
                for (int j = 0; j < 2 * r && cnt <= min_nb; j++, a++, b--, l -= TW, g += TW) {
                    test(*a);
                    test(*b);
                    test(*l);
                    test(*g);
                }
            }
            for (int i = -hw; WIDE && nr < hw && i <= hw && cnt <= min_nb; i++) {
                const float4* row = centre + i * TW;
                const bool split = i >= -nr && i <= nr;
                const int e = split ? -nr - 1 : hw;
                for (int j = -hw; j <= e; j++) test(row[j]);
                if (split)
                    for (int j = nr + 1; j <= hw; j++) test(row[j]);
            }
            keep = cnt > min_nb || (WIDE && min_nb <= 0);
        }
        const size_t o = (size_t)y * cols + x;
        out[3 * o] = keep ? c.x : 0.f;
        out[3 * o + 1] = keep ? c.y : 0.f;
        out[3 * o + 2] = keep ? c.z : 0.f;
        mask_out[o] = keep ? 1 : 0;
    }
    __syncthreads();
}

}  // namespace zt
