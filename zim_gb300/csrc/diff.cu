// diff.cu -- differentiable sub-pixel matching + reprojection: forward and
// hand-written adjoint w.r.t. the stereo calibration and the per-pixel phase.
//
// No counterpart in the reference (it has no gradients).  The forward follows
// its sub-pixel refinement and rectified-coordinate reprojection
// (PhaseShiftGrayCode3D/src/JSLAB_PhaseEpipolarReconstructor_V2.cpp:985-1000,
// :414-461) on rectified phase sampled with exact bilinear weights from the
// source phase through the undistort-rectify ray model of
// initUndistortRectifyMap (:329-337).  The match columns are inputs.
//
// Per rectified left pixel (j, i) with match column b:
//   phi_L = phase_L(map_L(j, i)),  phi_R,m = phase_R(map_R(b - 1 + m, i))
//   c_m = phi_R,m - phi_L;  delta = c1 (c0 - c2) / (2 (c0 - c1)(c1 - c2))
//   d = j - b - delta;  w = q32 d + q33;  P = (j + q03, i + q13, q23) / w
// Every parameter reaches P through the scalar w, so dP/dtheta = -P/w dw/dtheta:
// the kernel builds dw/dtheta (16 values) per point from the samples'
// position Jacobians and the phase slopes, then
//   dLoss/dtheta += -(g . P)/w * dw/dtheta   (g = upstream dLoss/dP)
//   J_r = -(n . P)/w * dw/dtheta             (plane distance, for J^T J).
// The loss is summed in FP64 per thread, the gradient as two-float sums, J^T J in
// FP32 over 32 points and then as two-float sums, normalised at every view's end; warps,
// blocks and their partials add in FP64 in a fixed order.
#include <cmath>
#include <cstring>
#include <vector>

#include "zim_internal.cuh"

namespace {

constexpr int DIFF_T = 128;   // threads per block
constexpr int DIFF_W = DIFF_T / 32;
constexpr int NP = ZIM_DIFF_NPARAMS;
constexpr int NJ = NP * (NP + 1) / 2;  // 136 upper-triangle entries of J^T J
constexpr int NACC = 2 + NP + NJ;       // loss, count, grad, jtj
constexpr int MAX_VIEWS = 4096;
// blocks per SM
constexpr int DIFF_FWD = 6, DIFF_BWD = 4, DIFF_UP = 3;

struct DiffCam {
    float ir[9];  // rectified pixel -> camera ray
    float fx, fy, cx, cy, k1, k2, p1, p2, k3;
};

struct DiffDev {
    DiffCam cam[2];
    float q03, q13, q23, q32, q33;
    double q03d, q13d, q23d, q32d, q33d;  // the same in FP64, for w and the plane distance
    float dq32, dq33;  // d/d baseline
    int rw, rh, sw, sh;
    float zmin, zmax;
};

struct ViewDev {
    const int32_t* order[2];
    const float* res[2];
    const int32_t* best;
    double nd[3], pdd;  // plane
    float* xyz;
    uint8_t* mask;
    const float* gxyz;
    float* gphase[2];
};

// One phase sample of camera cam at rectified (col, row): normalised ray (x, y),
// source pixel (x0, y0) + (a, b), bilinear phase base + frac (phase = 2 pi base +
// frac) and its slopes.  In three steps, so that a point's samples can be located
// first and all their taps loaded together.
struct Sample {
    int base, x0, y0;
    float frac, a, b, gu, gv, x, y;
};
struct Taps {
    int k[4];
    float r[4];
};

// False when a tap lies outside the image (also for NaN).
__device__ __forceinline__ bool locate(const DiffCam& c, float col, float row, int sw, int sh, Sample& s) {
    const float X0 = fmaf(c.ir[0], col, fmaf(c.ir[1], row, c.ir[2]));
    const float X1 = fmaf(c.ir[3], col, fmaf(c.ir[4], row, c.ir[5]));
    const float X2 = fmaf(c.ir[6], col, fmaf(c.ir[7], row, c.ir[8]));
    const float x = X0 / X2, y = X1 / X2;
    const float r2 = fmaf(x, x, y * y);
    const float sd = fmaf(r2, fmaf(r2, fmaf(r2, c.k3, c.k2), c.k1), 1.0f);
    const float xd = fmaf(x, sd, fmaf(2.0f * c.p1, x * y, c.p2 * fmaf(2.0f * x, x, r2)));
    const float yd = fmaf(y, sd, fmaf(c.p1, fmaf(2.0f * y, y, r2), 2.0f * c.p2 * x * y));
    const float u = fmaf(c.fx, xd, c.cx), v = fmaf(c.fy, yd, c.cy);
    const bool in = u >= 0.f && v >= 0.f && u < (float)(sw - 1) && v < (float)(sh - 1);
    s.x0 = (int)u;
    s.y0 = (int)v;
    s.a = u - (float)s.x0;
    s.b = v - (float)s.y0;
    s.x = x;
    s.y = y;
    return in && s.x0 + 1 < sw && s.y0 + 1 < sh;
}

__device__ __forceinline__ void load_taps(const int32_t* __restrict__ ord, const float* __restrict__ res, int sw,
                                          const Sample& s, bool in, Taps& t) {
    const size_t o = in ? (size_t)s.y0 * sw + s.x0 : 0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const size_t e = o + (q >> 1) * (size_t)sw + (q & 1);
        t.k[q] = in ? __ldg(ord + e) : 0;
        t.r[q] = in ? __ldg(res + e) : 0.f;
    }
}

// False when a tap is invalid (order < 1).
__device__ __forceinline__ bool interpolate(const Taps& t, Sample& s) {
    if (t.k[0] < 1 || t.k[1] < 1 || t.k[2] < 1 || t.k[3] < 1) return false;
    // phases relative to tap 00, integer cycles subtracted exactly
    const float p10 = fmaf((float)(t.k[1] - t.k[0]), ZIM_TWO_PI_F, t.r[1] - t.r[0]);
    const float p01 = fmaf((float)(t.k[2] - t.k[0]), ZIM_TWO_PI_F, t.r[2] - t.r[0]);
    const float p11 = fmaf((float)(t.k[3] - t.k[0]), ZIM_TWO_PI_F, t.r[3] - t.r[0]);
    const float a = s.a, b = s.b;
    s.base = t.k[0];
    s.frac = t.r[0] + fmaf(a * (1.0f - b), p10, fmaf((1.0f - a) * b, p01, a * b * p11));
    s.gu = fmaf(1.0f - b, p10, b * (p11 - p01));
    s.gv = fmaf(1.0f - a, p01, a * (p11 - p10));
    return true;
}

__device__ __forceinline__ bool take_sample(const DiffCam& c, float col, float row, const int32_t* __restrict__ ord,
                                            const float* __restrict__ res, int sw, int sh, Sample& s) {
    if (!locate(c, col, row, sw, sh, s)) return false;
    Taps t;
    load_taps(ord, res, sw, s, true, t);
    return interpolate(t, s);
}

// Adds to Jc (fx fy cx cy k1 k2) and, for the right camera, to Jrot what a sample
// of weight W = dw/dphi contributes to dw/dtheta: W (gu du/dtheta + gv dv/dtheta).
template <bool ROT>
__device__ __forceinline__ void add_jacobian(const DiffCam& c, const Sample& s, float W, float* Jc, float* Jrot) {
    const float x = s.x, y = s.y, gu = s.gu, gv = s.gv;
    const float r2 = fmaf(x, x, y * y);
    const float sd = fmaf(r2, fmaf(r2, fmaf(r2, c.k3, c.k2), c.k1), 1.0f);
    const float xd = fmaf(x, sd, fmaf(2.0f * c.p1, x * y, c.p2 * fmaf(2.0f * x, x, r2)));
    const float yd = fmaf(y, sd, fmaf(c.p1, fmaf(2.0f * y, y, r2), 2.0f * c.p2 * x * y));
    const float r4 = r2 * r2, fx = c.fx * x, fy = c.fy * y;
    Jc[0] = fmaf(W, __fmul_rn(gu, xd), Jc[0]);
    Jc[1] = fmaf(W, __fmul_rn(gv, yd), Jc[1]);
    Jc[2] = fmaf(W, gu, Jc[2]);
    Jc[3] = fmaf(W, gv, Jc[3]);
    Jc[4] = fmaf(W, fmaf(gu, fx * r2, __fmul_rn(gv, fy * r2)), Jc[4]);
    Jc[5] = fmaf(W, fmaf(gu, fx * r4, __fmul_rn(gv, fy * r4)), Jc[5]);
    if (ROT) {
        // ray X -> X + X x eps: d(x, y)/d eps_k for k = 0, 1, 2
        const float dx[3] = {x * y, -1.0f - x * x, y};
        const float dy[3] = {1.0f + y * y, -x * y, -x};
        const float s1 = fmaf(r2, fmaf(3.0f * c.k3, r2, 2.0f * c.k2), c.k1);  // d sd / d r2
        const float dxd_dx = sd + 2.0f * x * x * s1 + 2.0f * c.p1 * y + 6.0f * c.p2 * x;
        const float dxd_dy = 2.0f * x * y * s1 + 2.0f * c.p1 * x + 2.0f * c.p2 * y;
        const float dyd_dx = dxd_dy;
        const float dyd_dy = sd + 2.0f * y * y * s1 + 6.0f * c.p1 * y + 2.0f * c.p2 * x;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float ju = c.fx * fmaf(dxd_dx, dx[k], dxd_dy * dy[k]);
            const float jv = c.fy * fmaf(dyd_dx, dx[k], dyd_dy * dy[k]);
            Jrot[k] = fmaf(W, fmaf(gu, ju, __fmul_rn(gv, jv)), Jrot[k]);
        }
    }
}

__global__ void diff_rectify_kernel(DiffDev P, int cam, const int32_t* __restrict__ ord, const float* __restrict__ res,
                                    int32_t* __restrict__ rbase, float* __restrict__ rres,
                                    int32_t* __restrict__ rorder) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (j >= P.rw || i >= P.rh) return;
    Sample s;
    const size_t o = (size_t)i * P.rw + j;
    if (take_sample(P.cam[cam], (float)j, (float)i, ord, res, P.sw, P.sh, s)) {
        const int nx = s.a >= 0.5f ? s.x0 + 1 : s.x0, ny = s.b >= 0.5f ? s.y0 + 1 : s.y0;
        rbase[o] = s.base;
        rres[o] = s.frac;
        rorder[o] = __ldg(ord + (size_t)ny * P.sw + nx);
    } else {
        rbase[o] = 0;
        rres[o] = 0.f;
        rorder[o] = 0;
    }
}

__device__ __forceinline__ void scatter_phase(float* g, int sw, const Sample& s, float v) {
    if (!g || v == 0.f) return;
    const size_t o = (size_t)s.y0 * sw + s.x0;
    atomicAdd(g + o, v * (1.0f - s.a) * (1.0f - s.b));
    atomicAdd(g + o + 1, v * s.a * (1.0f - s.b));
    atomicAdd(g + o + sw, v * (1.0f - s.a) * s.b);
    atomicAdd(g + o + sw + 1, v * s.a * s.b);
}

// Sum of many FP32 values as an unevaluated pair of floats (Knuth's two-sum: the
// rounding error of each addition is added to lo).  The values are added as they
// are rounded: a product fused into the addition would not match its error term.
// An infinite sum has no error term (its lo is NaN).  lo's own roundings grow with it,
// so the pair is normalised now and then: 65536 terms of one sign (16 per view of 4096)
// ended up to 5e-8 off in a lane and 6e-11 in the total without, and are within what
// FP64 sums of as many terms guarantee (7e-12) with.  Over 704 values the error to the
// exact sum is that of FP64 sums of the same values (1.2e-10 of the sum of magnitudes,
// from the values' own rounding).  (Folding the pairs into FP64 every 63 points cost 9 %
// of the adjoint: two FP64 additions per clock and SM.)
struct Sum2 {
    float hi, lo;
    __device__ __forceinline__ void add(float v) {
        const float t = __fadd_rn(hi, v), z = __fsub_rn(t, hi);
        lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(t, z)), __fsub_rn(v, z)));
        hi = t;
    }
    // lo within half an ulp of hi again (Dekker's fast two-sum)
    __device__ __forceinline__ void normalise() {
        const float t = __fadd_rn(hi, lo);
        lo = __fsub_rn(lo, __fsub_rn(t, hi));
        hi = t;
    }
    __device__ __forceinline__ double value() const {
        return isfinite(hi) ? (double)hi + (double)lo : (double)hi;
    }
};

// The blocks of J^T J that are kept, 4 x 4 each: the ten on and above the diagonal.
constexpr int NBLK = 10;
constexpr int ROW = 20;  // floats per staged row of J (16 used): 16-byte loads without bank conflicts
__device__ __forceinline__ int block_row(int q) { return q < 4 ? 0 : q < 7 ? 1 : q < 9 ? 2 : 3; }
__device__ __forceinline__ int block_col(int q) { return q < 4 ? q : q < 7 ? q - 3 : q < 9 ? q - 5 : 3; }
// upper-triangle entry (a, b), a <= b, in row-major order
__device__ __forceinline__ int jtj_entry(int a, int b) { return a * NP - a * (a - 1) / 2 + b - a; }

// A thread per rectified left pixel of a view.  BWD: also J^T J and the gradient.
// UP: an upstream gradient of the points or a phase gradient is asked for.
//
// The gradient's FP32 terms add up as two-float sums (with an upstream gradient per
// thread, else through shared memory, lane k of a half-warp component k of the
// warp's points: two registers instead of 32).  J^T J: the rows of 3 x 32 points go
// through shared memory, and three groups of ten lanes each add up the ten blocks of
// 32 rows' outer products, 16 products per two 16-byte loads, in FP32 over the 32 and
// then as two-float sums.  (One product per two 4-byte loads, and 37 FP64 conversions
// and additions per 32 points, held the kernel at the FP64 and shared-memory pipes.)
// A point's four samples are located before any of their 32 loads, so that these are
// in flight together.  Four 2448x2048 views: 4.23 -> 1.18 ms; bound by issue and
// latency, with 16 warps per SM (12: 1.27), and the FP64 pipe half busy with the
// points' distances.
template <bool BWD, bool UP>
__global__ void __launch_bounds__(DIFF_T, BWD ? (UP ? DIFF_UP : DIFF_BWD) : DIFF_FWD)
    diff_kernel(const __grid_constant__ DiffDev P,
                                                         const ViewDev* __restrict__ views, int n_views,
                                                         float loss_weight, double* __restrict__ part) {
    __shared__ __align__(16) float rows[BWD ? DIFF_W : 1][3][32][ROW];
    __shared__ __align__(16) float terms[BWD && !UP ? DIFF_W : 1][32][ROW];
    __shared__ double red[DIFF_W][NACC];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const size_t npx = (size_t)P.rw * P.rh;
    const size_t nwarps = (size_t)gridDim.x * DIFF_W;
    double loss = 0.0;
    unsigned cnt = 0u;
    Sum2 g[UP ? NP : 1];
    Sum2 sum[16];
#pragma unroll
    for (int k = 0; k < (UP ? NP : 1); k++) g[k] = Sum2{0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 16; k++) sum[k] = Sum2{0.f, 0.f};
    const int grp = lane / NBLK, blk = lane - grp * NBLK;  // lanes 30 and 31 add up nothing
    const int br = 4 * block_row(blk), bc = 4 * block_col(blk);
    // adds the n staged sets of 32 rows, one per group of lanes
    int n_sets = 0;
    auto add_sets = [&]() {
        if (grp < n_sets) {
            float acc[16];
#pragma unroll
            for (int k = 0; k < 16; k++) acc[k] = 0.f;
#pragma unroll 4
            for (int p = 0; p < 32; p++) {
                const float4 u4 = *reinterpret_cast<const float4*>(&rows[wib][grp][p][br]);
                const float4 v4 = *reinterpret_cast<const float4*>(&rows[wib][grp][p][bc]);
                const float u[4] = {u4.x, u4.y, u4.z, u4.w}, v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
                for (int a = 0; a < 4; a++)
#pragma unroll
                    for (int e = 0; e < 4; e++) acc[4 * a + e] = fmaf(u[a], v[e], acc[4 * a + e]);
            }
#pragma unroll
            for (int k = 0; k < 16; k++) sum[k].add(acc[k]);
        }
        n_sets = 0;
    };

    // A warp strides over each view's pixels: the loop bound depends on the warp only,
    // so the lanes stay together, and (i, j) follow without divisions.  The sets of 32
    // pixels are those of all views' pixels in one row, whose first and last in a view
    // may be incomplete.
    const int stride = (int)nwarps * 32, di = stride / P.rw, dj = stride - di * P.rw;
    const size_t base0 = ((size_t)blockIdx.x * DIFF_W + wib) * 32;
    for (int vi = 0; vi < n_views; vi++) {
        const ViewDev& V = views[vi];
        const int shift = (int)(vi * npx & 31);
        size_t pix = base0 + lane - shift;  // wraps above npx for the shift's first lanes
        int i = (int)((base0 + lane - shift + 32 * (size_t)P.rw) / P.rw) - 32;
        int j = (int)(pix - (size_t)i * P.rw);
        int bnext = pix < npx ? __ldg(V.best + pix) : -1;
        for (size_t base = base0; base < npx + shift; base += stride, pix += stride) {
            float J[NP], s_r = 0.f, s_up = 0.f;
#pragma unroll
            for (int k = 0; k < NP; k++) J[k] = 0.f;
            const int b = bnext;
            bnext = pix + stride < npx ? __ldg(V.best + pix + stride) : -1;
            bool ok = pix < npx && b >= 1 && b + 1 < P.rw;
            Sample sL, sR[3];
            {
                Taps tL, tR[3];
                const bool l = ok && locate(P.cam[0], (float)j, (float)i, P.sw, P.sh, sL);
                bool in[3];
#pragma unroll
                for (int m = 0; m < 3; m++) in[m] = ok && locate(P.cam[1], (float)(b - 1 + m), (float)i, P.sw, P.sh, sR[m]);
                load_taps(V.order[0], V.res[0], P.sw, sL, l, tL);
#pragma unroll
                for (int m = 0; m < 3; m++) load_taps(V.order[1], V.res[1], P.sw, sR[m], in[m], tR[m]);
                ok = l && in[0] && in[1] && in[2] && interpolate(tL, sL);
#pragma unroll
                for (int m = 0; m < 3; m++) ok = ok && interpolate(tR[m], sR[m]);
            }
            float c[3] = {0.f, 0.f, 0.f};
            float delta = 0.f, dd[3] = {0.f, 0.f, 0.f};  // d delta / d c_m
            float X = 0.f, Y = 0.f, Z = 0.f, w = 0.f, d = 0.f;
            if (ok) {
#pragma unroll
                for (int m = 0; m < 3; m++) c[m] = fmaf((float)(sR[m].base - sL.base), ZIM_TWO_PI_F, sR[m].frac - sL.frac);
                const float num = c[1] * (c[0] - c[2]);
                const float den = 2.0f * (c[0] - c[1]) * (c[1] - c[2]);
                if (fabsf(den) > 1e-9f) {
                    delta = num / den;
                    const float inv = 1.0f / den;
                    dd[0] = (c[1] - delta * 2.0f * (c[1] - c[2])) * inv;
                    dd[1] = ((c[0] - c[2]) - delta * 2.0f * (c[0] - 2.0f * c[1] + c[2])) * inv;
                    dd[2] = (-c[1] + delta * 2.0f * (c[0] - c[1])) * inv;
                }
                d = (float)(j - b) - delta;
                ok = fabsf(d) >= 1e-5f;
            }
            // w from the exact integer part of the disparity and the FP32 sub-pixel
            // part: an FP32 disparity of ~1000 px would round at 6e-5 px
            double wd = 0.0;
            if (ok) {
                wd = fma(P.q32d, (double)(j - b) - (double)delta, P.q33d);
                w = (float)wd;
                if (fabsf(w) < 1e-2f * (fabsf(P.q32 * d) + fabsf(P.q33))) {
                    // near-zero disparity: the triangulation divide in FP64
                    X = (float)(((double)j + P.q03d) / wd);
                    Y = (float)(((double)i + P.q13d) / wd);
                    Z = (float)(P.q23d / wd);
                } else {
                    const float iw = 1.0f / w;
                    X = ((float)j + P.q03) * iw;
                    Y = ((float)i + P.q13) * iw;
                    Z = P.q23 * iw;
                }
                ok = Z > P.zmin && Z < P.zmax && isfinite(X) && isfinite(Y);
            }
            if (!BWD && pix < npx) {
                if (V.xyz) {
                    V.xyz[3 * pix] = ok ? X : 0.f;
                    V.xyz[3 * pix + 1] = ok ? Y : 0.f;
                    V.xyz[3 * pix + 2] = ok ? Z : 0.f;
                }
                if (V.mask) V.mask[pix] = ok ? 1 : 0;
            }
            if (ok) {
                // plane distance r = n . P + d = N / w, N = n . (j + q03, i + q13, q23) + d w
                // in FP64: the terms are ~1e3 times r, FP32 would lose three digits
                const double Nd = fma(V.nd[0], (double)j + P.q03d,
                                      fma(V.nd[1], (double)i + P.q13d, fma(V.nd[2], P.q23d, V.pdd * wd)));
                const float iw = 1.0f / w;
                const float r = (float)Nd * iw;
                loss += (double)r * (double)r;
                cnt++;
                if (BWD) {
                    // n . P = r - d, and dr/dw = -(n . P)/w
                    const float nP = r - (float)V.pdd;
                    s_r = -nP * iw;
                    // dw/dphi: d = j - b - delta, w = q32 d + q33
                    const float wR[3] = {-P.q32 * dd[0], -P.q32 * dd[1], -P.q32 * dd[2]};
                    const float wL = -(wR[0] + wR[1] + wR[2]);
                    J[12] = fmaf(d, P.dq32, P.dq33);
                    add_jacobian<false>(P.cam[0], sL, wL, J, nullptr);
#pragma unroll
                    for (int m = 0; m < 3; m++) add_jacobian<true>(P.cam[1], sR[m], wR[m], J + 6, J + 13);
                    // dLoss/dw = -(g . P)/w with g = lw 2 r n + grad_xyz
                    float gP = loss_weight * 2.0f * r * nP;
                    if (UP && V.gxyz)
                        gP += fmaf(V.gxyz[3 * pix], X, fmaf(V.gxyz[3 * pix + 1], Y, V.gxyz[3 * pix + 2] * Z));
                    s_up = -gP * iw;
                    if (UP) {
                        scatter_phase(V.gphase[0], P.sw, sL, s_up * wL);
#pragma unroll
                        for (int m = 0; m < 3; m++) scatter_phase(V.gphase[1], P.sw, sR[m], s_up * wR[m]);
                    }
#pragma unroll
                    for (int k = 0; k < NP; k++)
                        if (UP) g[k].add(__fmul_rn(s_up, J[k]));
                }
            }
            if (BWD) {
                // dLoss/dw J_w and the row of J_r = dr/dw J_w (0 where there is no point)
                float4* row = reinterpret_cast<float4*>(rows[wib][n_sets][lane]);
#pragma unroll
                for (int k = 0; k < NP; k += 4) {
                    if (!UP)
                        reinterpret_cast<float4*>(terms[wib][lane])[k / 4] =
                            make_float4(s_up * J[k], s_up * J[k + 1], s_up * J[k + 2], s_up * J[k + 3]);
                    row[k / 4] = make_float4(s_r * J[k], s_r * J[k + 1], s_r * J[k + 2], s_r * J[k + 3]);
                }
                n_sets++;
                __syncwarp();
                if (!UP) {
                    // lane k of each half-warp: component k over half of the rows (those
                    // apart by four, whose words lie in other banks)
#pragma unroll 4
                    for (int p = 0; p < 16; p++)
                        g[0].add(terms[wib][(p & 3) | (p & 12) << 1 | (lane & 16) >> 2][lane & 15]);
                }
                if (n_sets == 3) {
                    add_sets();
                    if (!UP) g[0].normalise();
                }
                __syncwarp();
            }
            i += di;
            j += dj;
            if (j >= P.rw) {
                j -= P.rw;
                i++;
            }
        }
        if (BWD) {
#pragma unroll
            for (int k = 0; k < (UP ? NP : 0); k++) g[k].normalise();
#pragma unroll
            for (int k = 0; k < 16; k++) sum[k].normalise();
        }
    }
    // warp sums (fixed shuffle tree), then per-warp rows summed in warp order
    double dcnt = (double)cnt;
    for (int off = 16; off; off >>= 1) {
        loss += __shfl_xor_sync(0xffffffffu, loss, off);
        dcnt += __shfl_xor_sync(0xffffffffu, dcnt, off);
    }
    if (lane == 0) {
        red[wib][0] = loss;
        red[wib][1] = dcnt;
    }
    if (BWD) {
#pragma unroll
        for (int k = 0; k < (UP ? NP : 1); k++) {
            double v = g[k].value();
            for (int off = 16; off >= (UP ? 1 : 16); off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if (UP && lane == 0) red[wib][2 + k] = v;
            if (!UP && lane < NP) red[wib][2 + lane] = v;
        }
        add_sets();
#pragma unroll
        for (int k = 0; k < 16; k++) {
            double v = sum[k].value();
            // the three groups' shares of the rows
            const double v1 = __shfl_down_sync(0xffffffffu, v, NBLK), v2 = __shfl_down_sync(0xffffffffu, v, 2 * NBLK);
            v = (v + v1) + v2;
            const int a = br + k / 4, e = bc + k % 4;
            if (lane < NBLK && a <= e) red[wib][2 + NP + jtj_entry(a, e)] = v;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < (BWD ? NACC : 2); e += DIFF_T) {
        double s = 0.0;
        for (int ww = 0; ww < DIFF_W; ww++) s += red[ww][e];
        part[(size_t)blockIdx.x * NACC + e] = s;
    }
}

// Fixed-order sum of the block partials: a warp per accumulator.
__global__ void diff_total_kernel(const double* __restrict__ part, int nblk, int n, double* __restrict__ out) {
    const int e = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (e >= n) return;
    double s = 0.0;
    for (int b = lane; b < nblk; b += 32) s += part[(size_t)b * NACC + e];
    for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) out[e] = s;
}

// Rotation matrix of a rotation vector (Rodrigues' formula), row-major.
void rodrigues(const double v[3], double R[9]) {
    const double th = std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    double k[3] = {0, 0, 0}, c = 1.0, s = 0.0, cc = 0.0;
    if (th > 0) {
        for (int a = 0; a < 3; a++) k[a] = v[a] / th;
        c = std::cos(th);
        s = std::sin(th);
        cc = 1.0 - c;
    }
    R[0] = c + cc * k[0] * k[0];        R[1] = cc * k[0] * k[1] - s * k[2]; R[2] = cc * k[0] * k[2] + s * k[1];
    R[3] = cc * k[1] * k[0] + s * k[2]; R[4] = c + cc * k[1] * k[1];        R[5] = cc * k[1] * k[2] - s * k[0];
    R[6] = cc * k[2] * k[0] - s * k[1]; R[7] = cc * k[2] * k[1] + s * k[0]; R[8] = c + cc * k[2] * k[2];
}

zim_status make_dev(zim_ctx* ctx, const zim_diff_params* p, double zmin, double zmax, DiffDev& D) {
    if (!ctx->calibrated) return zim_fail(ctx, ZIM_ERR_NOT_CALIBRATED, "not calibrated");
    const double* t = ctx->calib.t;
    const double B0 = std::sqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
    if (!(p->baseline > 0) || !(B0 > 0)) return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "baseline must be > 0");
    for (int c = 0; c < 2; c++) {
        DiffCam& C = D.cam[c];
        double ir[9];
        if (c == 0) {
            std::memcpy(ir, ctx->ir[0], sizeof ir);
        } else {
            // (P2' R2 E)^-1 = E^T (P2' R2)^-1
            double E[9];
            rodrigues(p->rot, E);
            for (int r = 0; r < 3; r++)
                for (int q = 0; q < 3; q++) {
                    double s = 0;
                    for (int m = 0; m < 3; m++) s += E[m * 3 + r] * ctx->ir[1][m * 3 + q];
                    ir[r * 3 + q] = s;
                }
        }
        for (int a = 0; a < 9; a++) C.ir[a] = (float)ir[a];
        C.fx = (float)p->cam[c][0]; C.fy = (float)p->cam[c][1];
        C.cx = (float)p->cam[c][2]; C.cy = (float)p->cam[c][3];
        C.k1 = (float)p->cam[c][4]; C.k2 = (float)p->cam[c][5];
        const double* Dc = ctx->calib.dist_coeffs[c];
        C.p1 = (float)Dc[2]; C.p2 = (float)Dc[3]; C.k3 = (float)Dc[4];
    }
    const double* Q = ctx->Q;
    const double Tx0 = -1.0 / Q[14], dcx = Q[15] * Tx0;
    const double Tx = Tx0 * p->baseline / B0, dTx = Tx0 / B0;
    D.q03d = Q[3]; D.q13d = Q[7]; D.q23d = Q[11];
    D.q32d = -1.0 / Tx;
    D.q33d = dcx / Tx;
    D.q03 = (float)Q[3]; D.q13 = (float)Q[7]; D.q23 = (float)Q[11];
    D.q32 = (float)(-1.0 / Tx);
    D.q33 = (float)(dcx / Tx);
    D.dq32 = (float)(dTx / (Tx * Tx));
    D.dq33 = (float)(-dcx * dTx / (Tx * Tx));
    D.rw = ctx->rect_w; D.rh = ctx->rect_h; D.sw = ctx->src_w; D.sh = ctx->src_h;
    D.zmin = (float)zmin; D.zmax = (float)zmax;
    return ZIM_OK;
}

zim_status run(zim_ctx* ctx, const zim_diff_params* params, const zim_diff_view* views, int n_views, int rows,
               int cols, double zmin, double zmax, bool bwd, double loss_weight, zim_diff_result* out, void* stream) {
    if (!ctx) return ZIM_ERR_INVALID_ARG;
    if (!params || !views || !out || n_views < 1 || n_views > MAX_VIEWS)
        return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "bad argument (n_views must be in [1, %d])", MAX_VIEWS);
    DiffDev D;
    zim_status s = make_dev(ctx, params, zmin, zmax, D);
    if (s) return s;
    if (rows != ctx->src_h || cols != ctx->src_w)
        return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "phase size %dx%d differs from the calibration's %dx%d", cols, rows,
                        ctx->src_w, ctx->src_h);
    std::vector<ViewDev> hv((size_t)n_views);
    for (int v = 0; v < n_views; v++) {
        const zim_diff_view& V = views[v];
        if (!V.order[0] || !V.order[1] || !V.residual[0] || !V.residual[1] || !V.best_col)
            return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "view %d: missing phase or match columns", v);
        ViewDev& H = hv[(size_t)v];
        for (int c = 0; c < 2; c++) {
            H.order[c] = V.order[c];
            H.res[c] = V.residual[c];
            H.gphase[c] = bwd ? V.grad_phase[c] : nullptr;
        }
        H.best = V.best_col;
        for (int a = 0; a < 3; a++) H.nd[a] = V.plane[a];
        H.pdd = V.plane[3];
        H.xyz = bwd ? nullptr : V.xyz;
        H.mask = bwd ? nullptr : V.mask;
        H.gxyz = bwd ? V.grad_xyz : nullptr;
    }
    bool up = false;  // an upstream gradient, or phase gradients
    for (const ViewDev& H : hv) up = up || H.gxyz || H.gphase[0] || H.gphase[1];
    // all blocks resident at once
    const int nblk = (!bwd ? DIFF_FWD : up ? DIFF_UP : DIFF_BWD) * (ctx->sm_count > 0 ? ctx->sm_count : 152);
    zim_scratch_reset(ctx);
    s = zim_scratch_reserve(ctx, zim_align256(hv.size() * sizeof(ViewDev)) + zim_align256((size_t)nblk * NACC * 8) +
                                     zim_align256(NACC * 8) + 4096);
    if (s) return s;
    ViewDev* dv = (ViewDev*)zim_scratch_take(ctx, hv.size() * sizeof(ViewDev));
    double* part = (double*)zim_scratch_take(ctx, (size_t)nblk * NACC * 8);
    double* tot = (double*)zim_scratch_take(ctx, NACC * 8);
    cudaStream_t st = zim_stream(stream);
    static_assert(NACC * 8 <= 4096, "totals fit the pinned staging");
    ZIM_CUDA_TRY(ctx, cudaMemcpyAsync(dv, hv.data(), hv.size() * sizeof(ViewDev), cudaMemcpyHostToDevice, st));
    auto kern = !bwd ? diff_kernel<false, false> : up ? diff_kernel<true, true> : diff_kernel<true, false>;
    kern<<<nblk, DIFF_T, 0, st>>>(D, dv, n_views, (float)loss_weight, part);
    const int n = bwd ? NACC : 2;
    diff_total_kernel<<<(n + 7) / 8, 256, 0, st>>>(part, nblk, n, tot);
    ctx->launches += 2;
    ZIM_LAUNCH_CHECK(ctx);
    double* h = (double*)ctx->h_pinned;
    ZIM_CUDA_TRY(ctx, cudaMemcpyAsync(h, tot, NACC * 8, cudaMemcpyDeviceToHost, st));
    ZIM_CUDA_TRY(ctx, cudaStreamSynchronize(st));
    std::memset(out, 0, sizeof *out);
    out->loss = h[0];
    out->n_points = h[1];
    if (bwd) {
        for (int k = 0; k < NP; k++) out->grad[k] = h[2 + k];
        int e = 0;
        for (int a = 0; a < NP; a++)
            for (int b = a; b < NP; b++, e++) out->jtj[a * NP + b] = out->jtj[b * NP + a] = h[2 + NP + e];
    }
    return ZIM_OK;
}

}  // namespace

extern "C" ZIM_API zim_status zim_diff_params_nominal(const zim_ctx* ctx, zim_diff_params* out) {
    if (!ctx || !out) return ZIM_ERR_INVALID_ARG;
    if (!ctx->calibrated) return ZIM_ERR_NOT_CALIBRATED;
    for (int c = 0; c < 2; c++) {
        const double* K = ctx->calib.camera_matrix[c];
        const double* D = ctx->calib.dist_coeffs[c];
        out->cam[c][0] = K[0]; out->cam[c][1] = K[4]; out->cam[c][2] = K[2]; out->cam[c][3] = K[5];
        out->cam[c][4] = D[0]; out->cam[c][5] = D[1];
    }
    const double* t = ctx->calib.t;
    out->baseline = std::sqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
    out->rot[0] = out->rot[1] = out->rot[2] = 0.0;
    return ZIM_OK;
}

extern "C" ZIM_API zim_status zim_diff_rectify(zim_ctx* ctx, const zim_diff_params* params, int cam,
                                               const int32_t* order, const float* residual, int rows, int cols,
                                               int32_t* rect_base, float* rect_res, int32_t* rect_order,
                                               void* stream) {
    if (!ctx) return ZIM_ERR_INVALID_ARG;
    if (!params || (cam != 0 && cam != 1) || !order || !residual || !rect_base || !rect_res || !rect_order)
        return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "bad argument");
    DiffDev D;
    zim_status s = make_dev(ctx, params, 0.0, 0.0, D);
    if (s) return s;
    if (rows != ctx->src_h || cols != ctx->src_w)
        return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "phase size %dx%d differs from the calibration's %dx%d", cols, rows,
                        ctx->src_w, ctx->src_h);
    dim3 grd((D.rw + 255) / 256, D.rh);
    diff_rectify_kernel<<<grd, 256, 0, zim_stream(stream)>>>(D, cam, order, residual, rect_base, rect_res,
                                                              rect_order);
    ctx->launches += 1;
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}

extern "C" ZIM_API zim_status zim_diff_forward(zim_ctx* ctx, const zim_diff_params* params,
                                               const zim_diff_view* views, int n_views, int rows, int cols,
                                               double z_min, double z_max, zim_diff_result* out, void* stream) {
    return run(ctx, params, views, n_views, rows, cols, z_min, z_max, false, 0.0, out, stream);
}

extern "C" ZIM_API zim_status zim_diff_backward(zim_ctx* ctx, const zim_diff_params* params,
                                                const zim_diff_view* views, int n_views, int rows, int cols,
                                                double z_min, double z_max, double loss_weight,
                                                zim_diff_result* out, void* stream) {
    return run(ctx, params, views, n_views, rows, cols, z_min, z_max, true, loss_weight, out, stream);
}
