// decode.cu -- per-pixel N-step phase-shift decode: fused 3x3 pre-blur,
// wrapped phase (atan2) + normalised modulation with the validity threshold,
// then heterodyne (reference), hierarchical or Gray-code unwrapping.
//
// Reference: PhaseShiftGrayCode3D/src/JSLAB_PhaseShiftDecoder_V2.cpp:18-28
// (pre-blur), :54-182 (decode body); GPU port JSLAB_PhaseShiftDecoder_V2_GPU.cu:44-146.
//
// Arithmetic is FP32.  The pre-blur is linear, so the blurred sums
// S = -sum sin_k I_k, C = sum cos_k I_k, sum I_k are the 3x3 blur of the raw
// per-pixel sums: 3 channels per frequency are blurred instead of N frames.
// Unwrapping keeps integer cycle counts exact and only small fractional parts
// in FP32, so an order differs from the FP64 restatement only when a decision
// argument sits within ~1e-6 of its threshold.
#include <cmath>
#include <mutex>
#include <type_traits>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "zim_tiles.cuh"

namespace {

using zt::DecodeParams;

constexpr int MAX_PS = 4;       // phase-shift frequencies
constexpr int DEC_WARPS = 4;    // warps per block
constexpr int STRIP = 30;       // output columns per warp (32 read)
constexpr int DEC_MIN_WARPS = 24;  // warps per SM a launch should have

__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }

// The two samples of a packed word as floats: each sample's bits under the
// exponent of 2^23, minus 2^23 (exact, no integer-to-float conversion).
template <typename T>
__device__ __forceinline__ float2 unpack(unsigned w) {
    const unsigned a = sizeof(T) == 2 ? __byte_perm(w, 0x4B000000u, 0x7410) : __byte_perm(w, 0x4B000000u, 0x7440);
    const unsigned b = sizeof(T) == 2 ? __byte_perm(w, 0x4B000000u, 0x7432) : __byte_perm(w, 0x4B000000u, 0x7441);
    return __fadd2_rn(make_float2(__uint_as_float(a), __uint_as_float(b)), both(-8388608.f));
}

// A lane's pixel pair of one row as a packed word: the second sample lies d (0
// or 1) after the first; PAIR: one aligned load of both.
template <typename T, bool PAIR>
__device__ __forceinline__ unsigned load_pair(const T* q, int d) {
    if (PAIR)
        return sizeof(T) == 2 ? __ldg(reinterpret_cast<const unsigned*>(q))
                              : (unsigned)__ldg(reinterpret_cast<const unsigned short*>(q));
    return (unsigned)__ldg(q) | (unsigned)__ldg(q + d) << (8 * sizeof(T));
}

// n words of consecutive frames (npx samples apart) from q on; the choice of load
// is the warp's (pair: every lane's pair is aligned and inside the image), so it
// costs one branch, not two loads in the place of each.
template <typename T, int N>
__device__ __forceinline__ void load_pairs(const T* q, size_t npx, bool pair, int d, unsigned (&w)[N]) {
    if (pair) {
#pragma unroll
        for (int k = 0; k < N; k++) w[k] = load_pair<T, true>(q + k * npx, d);
    } else {
#pragma unroll
        for (int k = 0; k < N; k++) w[k] = load_pair<T, false>(q + k * npx, d);
    }
}

// floor(a / b) for b > 0 and |a / b| < 2^21, from the float reciprocal
// inv_b = 1 / b: the float quotient is within one of the true one, and one
// remainder check corrects it (an integer division costs ~40 instructions).
__device__ __forceinline__ int floor_div(int a, int b, float inv_b) {
    int q = __float2int_rd((float)a * inv_b);
    const int r = a - q * b;
    q += (r >= b) - (r < 0);
    return q;
}

// The validity test on the normalised modulation nm = (2 |S, C| / N) / (M / N)
// (0 when M <= 1e-3 N): nm < thr fails the pixel.  For M > 0 that is
// 4 (S^2 + C^2) < (thr M)^2 with thr > 0, which needs neither the square root
// nor the division; they are computed only where nm is written out
// (want_value: frequency 0 with a modulation map).  The two forms decide
// differently only where nm lies within float rounding of thr.
__device__ __forceinline__ bool modulation_ok(float S, float C, float M, int N, float thr, bool want_value,
                                              float& value) {
    const float q = fmaf(S, S, C * C);
    const bool has_m = M > 1e-3f * (float)N;
    if (want_value) value = has_m ? 2.0f * sqrtf(q) / M : 0.f;
    if (!(thr > 0.f)) return true;
    const float tm = thr * M;
    return has_m && !(4.0f * q < tm * tm);
}

// Absolute order k and residual r of one pixel from its wrapped phases; g1, g2:
// its Gray codeword and, with the complementary bit, the shifted one.
template <int NPS>
__device__ __forceinline__ void unwrap(const DecodeParams& p, int n_ps, const float (&w)[MAX_PS], int g1, int g2,
                                       int& k, float& r) {
    k = 0;
    if (p.enc == ZIM_ENC_HETERODYNE3) {
        const float w0 = w[0], w1 = w[1], w2 = w[2];
        float p12 = w0 > w1 ? w0 - w1 : w0 - w1 + ZIM_TWO_PI_F;
        float p23;
        if (p.f1_gt_f2) p23 = w1 > w2 ? w1 - w2 : w1 - w2 + ZIM_TWO_PI_F;
        else p23 = w2 > w1 ? w2 - w1 : w2 - w1 + ZIM_TWO_PI_F;
        float p123 = p12 > p23 ? p12 - p23 : p12 - p23 + ZIM_TWO_PI_F;
        // uphase12 = p12 + 2 pi m12;  k = round(m12 f0 / f12 + (p12 f0 / f12 - w0) / 2 pi)
        int m12 = (int)roundf(fmaf(p123, (float)p.f12, -p12) * ZIM_INV_TWO_PI_F);
        int num = m12 * p.f0;
        int q = floor_div(num, p.f12, p.inv_f12);
        int rem = num - q * p.f12;
        k = q + (int)roundf(fmaf((float)rem, p.inv_f12, fmaf(p12, p.f0_f12, -w0) * ZIM_INV_TWO_PI_F));
        r = w0;
        if (p.avg3) {
            int m23 = (int)roundf(fmaf(p123, (float)p.f23, -p23) * ZIM_INV_TWO_PI_F);
            int n2 = m23 * p.f1, q2 = floor_div(n2, p.f23, p.inv_f23), r2i = n2 - q2 * p.f23;
            int k2 = q2 + (int)roundf(fmaf((float)r2i, p.inv_f23, fmaf(p23, p.f1_f23, -w1) * ZIM_INV_TWO_PI_F));
            int n3 = m23 * p.f2, q3 = floor_div(n3, p.f23, p.inv_f23), r3i = n3 - q3 * p.f23;
            int k3 = q3 + (int)roundf(fmaf((float)r3i, p.inv_f23, fmaf(p23, p.f2_f23, -w2) * ZIM_INV_TWO_PI_F));
            // (uphase2 f0 / f1 - 2 pi k) = (w1 f0 + 2 pi (k2 f0 - k f1)) / f1, same for 3
            float r2 = fmaf((float)(k2 * p.f0 - k * p.f1), ZIM_TWO_PI_F, w1 * (float)p.f0) * p.inv_f1;
            float r3 = fmaf((float)(k3 * p.f0 - k * p.f2), ZIM_TWO_PI_F, w2 * (float)p.f0) * p.inv_f2;
            r = (w0 + r2 + r3) * (1.0f / 3.0f);
        }
    } else if (p.enc == ZIM_ENC_HIERARCHICAL) {
        r = w[0];
#pragma unroll
        for (int i = 1; i < NPS; i++) {
            if (i >= n_ps) break;
            float a = fmaf(p.fratio[i], w[i - 1] + ZIM_PI_F, -(w[i] + ZIM_PI_F)) * ZIM_INV_TWO_PI_F;
            k = p.iratio[i] * k + (int)roundf(a);
            r = w[i];
        }
    } else {
        k = g1;
        r = w[0];
        if (p.complementary) {
            if (r <= -0.5f * ZIM_PI_F) k = g2;
            else if (r >= 0.5f * ZIM_PI_F) k = g2 - 1;
        }
    }
}

struct Outputs {
    int32_t* order;
    float* residual;
    float* mod;
    uint8_t* valid;
};
// The one or two cameras of a launch, one per blockIdx.y: the cameras of a small
// pair together fill the GPU, and a large pair has one last wave less (a whole pair
// with SOR, hierarchical: 99 -> 93 us at 640 x 480, 188 -> 181 at 1280 x 1024, 507 ->
// 500 at 2448 x 2048).  A single camera has a kernel of its own: its frames' base is
// then a constant of the launch (24 frames: 117 us; 127 without).
struct Cameras {
    const void* frames[2];
    Outputs out[2];
};

// A pixel under way: wrapped phases, modulation of frequency 0, whether nothing
// rejected it so far.
struct Pixel {
    float w[MAX_PS], mod;
    bool ok;
};

// One frequency's blurred (or fitted) sums: wrapped phase and validity.
__device__ __forceinline__ void take_frequency(const DecodeParams& p, int i, float S, float C, float M, bool want_mod,
                                               Pixel& px) {
    px.w[i] = zt::phase_atan2(S, C);
    float v = 0.f;
    const bool m = modulation_ok(S, C, M, p.shift[i], p.thr, want_mod && i == 0, v);
    if (i == 0) px.mod = px.ok ? v : 0.f;
    px.ok = px.ok && m;
}

// Unwraps and writes a pixel.
template <int NPS>
__device__ __forceinline__ void finish_pixel(const DecodeParams& p, int n_ps, const Pixel& px, int g1, int g2,
                                             size_t o, const Outputs& out) {
    int k;
    float r;
    unwrap<NPS>(p, n_ps, px.w, g1, g2, k, r);
    out.order[o] = px.ok ? k : (p.hdr ? -1 : 0);  // the HDR decoder marks invalid orders -1
    out.residual[o] = px.ok ? r : 0.f;
    if (out.mod) out.mod[o] = px.mod;
    if (out.valid) out.valid[o] = px.ok;
}

// One warp decodes a strip of 30 columns (a lane per column, one more on either
// side), marching down `band` rows: each raw row's sums are formed once,
// exchanged with the neighbour lanes by shuffles and added to the three output
// rows they blur into, so nothing is staged in shared memory and no warp waits
// for another.  The next row's samples are in flight while a row is blurred and
// unwrapped.  S and C are the lanes of the paired FP32 FMA (__ffma2_rn: each
// rounded as fmaf).  NS: frames per frequency; NPS: frequencies (no Gray code).
//
// Bound by instruction issue.  A tile (decode_tile_kernel: nine two-word shared loads
// per pixel and frequency, a 1.33x halo) issues 588 warp instructions per 32 pixels
// for three frequencies of four frames; this kernel issues 434.  Two columns per lane
// (all sums paired, half the shuffles) issued 409 but needed 120 registers and took 88
// us where this takes 73 (2448x2048, 12 16-bit frames; tiles 83).
template <typename T, int NPS, int NS>
__device__ __forceinline__ void decode_strip(const T* __restrict__ frames, const DecodeParams& p, int band, int nstrips,
                                             const Outputs& out) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int wid = blockIdx.x * DEC_WARPS + (threadIdx.x >> 5);
    const int y0 = (wid / nstrips) * band;
    if (y0 >= p.rows) return;
    const int y1 = min(y0 + band, p.rows);
    const int x = (wid % nstrips) * STRIP - 1 + lane;
    const bool writes = lane > 0 && lane < 31 && x < p.cols;
    const size_t npx = (size_t)p.rows * p.cols;
    // byte offset of a row's sample within any frame's plane (at most 2^31 samples):
    // the plane's base is the same for the whole grid, so a load adds 32 bits to it
    const int xc = min(max(x, 0), p.cols - 1);
    auto row_off = [&](int y) {
        return ((unsigned)min(max(y, 0), p.rows - 1) * (unsigned)p.cols + (unsigned)xc) * (unsigned)sizeof(T);
    };
    auto sample = [&](int f, unsigned off) {
        return (unsigned)__ldg(reinterpret_cast<const T*>(reinterpret_cast<const char*>(frames + (size_t)f * npx) + off));
    };
    constexpr int NW = NPS * NS;
    unsigned raw[NW];  // samples in flight
    auto fetch = [&](int y) {
        const unsigned o = row_off(y);
#pragma unroll
        for (int f = 0; f < NW; f++) raw[f] = sample(f, o);
    };
    // blurred sums under way: A for the row above the current raw row, B for it
    float2 A[NPS], B[NPS];  // (S, C)
    float AM[NPS], BM[NPS];
#pragma unroll
    for (int i = 0; i < NPS; i++) {
        A[i] = B[i] = make_float2(0.f, 0.f);
        AM[i] = BM[i] = 0.f;
    }
    fetch(y0 - 1);
    for (int y = y0 - 1; y <= y1; y++) {
        float2 sc[NPS];
        float m[NPS];
#pragma unroll
        for (int i = 0; i < NPS; i++) {
            sc[i] = make_float2(0.f, 0.f);
            auto add = [&](int f, unsigned w) {
                const float v = (float)w;
                sc[i] = make_float2(fmaf(-p.sinv[f], v, sc[i].x), fmaf(p.cosv[f], v, sc[i].y));
                m[i] += v;
            };
            sc[i].y = m[i] = (float)raw[i * NS];  // step 0: sin 0 and cos 1 exactly
#pragma unroll
            for (int k = 1; k < NS; k++) add(i * NS + k, raw[i * NS + k]);
        }
        if (y < y1) fetch(y + 1);
        Pixel px;
        px.ok = true;
#pragma unroll
        for (int i = 0; i < NPS; i++) {
            // taps in row-major order from zero, as nine sequential FMAs per output
            auto w2 = [&](int t) { return make_float2(p.w2d[t], p.w2d[t]); };
            const float2 c = sc[i];
            const float2 l = make_float2(__shfl_up_sync(full, c.x, 1), __shfl_up_sync(full, c.y, 1));
            const float2 r = make_float2(__shfl_down_sync(full, c.x, 1), __shfl_down_sync(full, c.y, 1));
            const float2 F = __ffma2_rn(w2(8), r, __ffma2_rn(w2(7), c, __ffma2_rn(w2(6), l, A[i])));
            A[i] = __ffma2_rn(w2(5), r, __ffma2_rn(w2(4), c, __ffma2_rn(w2(3), l, B[i])));
            B[i] = __ffma2_rn(w2(2), r, __ffma2_rn(w2(1), c, __ffma2_rn(w2(0), l, make_float2(0.f, 0.f))));
            const float ml = __shfl_up_sync(full, m[i], 1), mr = __shfl_down_sync(full, m[i], 1);
            const float FM = fmaf(p.w2d[8], mr, fmaf(p.w2d[7], m[i], fmaf(p.w2d[6], ml, AM[i])));
            AM[i] = fmaf(p.w2d[5], mr, fmaf(p.w2d[4], m[i], fmaf(p.w2d[3], ml, BM[i])));
            BM[i] = fmaf(p.w2d[2], mr, fmaf(p.w2d[1], m[i], fmaf(p.w2d[0], ml, 0.f)));
            if (y > y0) take_frequency(p, i, F.x, F.y, FM, out.mod != nullptr, px);
        }
        if (y > y0 && writes) finish_pixel<NPS>(p, NPS, px, 0, 0, (size_t)(y - 1) * p.cols + x, out);
    }
}
template <typename T, int NPS, int NS>
__global__ void __launch_bounds__(32 * DEC_WARPS) decode_strip_kernel(const T* __restrict__ frames,
                                                                      const __grid_constant__ DecodeParams p, int band,
                                                                      int nstrips, const __grid_constant__ Outputs out) {
    decode_strip<T, NPS, NS>(frames, p, band, nstrips, out);
}
template <typename T, int NPS, int NS>
__global__ void __launch_bounds__(32 * DEC_WARPS) decode_strips_kernel(const __grid_constant__ Cameras cams,
                                                                       const __grid_constant__ DecodeParams p, int band,
                                                                       int nstrips) {
    decode_strip<T, NPS, NS>(static_cast<const T*>(cams.frames[blockIdx.y]), p, band, nstrips, cams.out[blockIdx.y]);
}

// ------------------------------------------------------------------ tiles --
// A block decodes 32 x 8 pixels: the raw sums of the tile and its 1-pixel halo go
// to shared memory, each frequency's three channels are blurred from there.  NPS /
// NS: frequencies and frames per frequency at compile time (0: from p).  TMA: the
// phase-shift samples come in one bulk tensor copy (cp.async.bulk.tensor) completing
// on an mbarrier, from a 3-D map over (x, y, frame) of the frame stack; box BW x HY x
// nfr, its x XPAD pixels left of the tile (a copy's x must be 16-byte aligned), its y
// one row above.  Samples outside the image read as 0 and are never used: the sums
// clamp to the image.  All forms add in the strips' order, so the bits are the same.
//
// The loads of a tile are all in flight at once whatever the step count, where a
// strip keeps one row ahead and only a step count known at compile time can be held
// in registers, and a small image has its latency once instead of once a row.  Times
// of tiles / strips are at the rule (use_strips).
constexpr int TX = 32, TY = 8, HX = TX + 2, HY = TY + 2;
template <typename T>
__host__ __device__ constexpr int tma_xpad() { return 16 / (int)sizeof(T); }
template <typename T>
__host__ __device__ constexpr int tma_bw() { return TX + 2 * tma_xpad<T>(); }
constexpr int TMA_MAX_FRAMES = 24;           // box depth (phase-shift frames) the copy takes
constexpr unsigned TMA_POLLS = 1u << 22;     // mbarrier polls before giving up (well over a second)
constexpr uint32_t ERR_DECODE_COPY = 0x20u;  // device error word: a tile's copy did not land

struct TileMaps {
    CUtensorMap m[2];  // per camera
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Phase 0 of the barrier completed; false after `polls` polls.
__device__ __forceinline__ bool mbar_wait0(unsigned bar, unsigned polls) {
    for (unsigned it = 0; it < polls; it++) {
        unsigned done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(bar)
            : "memory");
        if (done) return true;
    }
    return false;
}

template <typename T, int NPS, int NS, bool TMA>
__global__ void __launch_bounds__(TX* TY) decode_tile_kernel(const __grid_constant__ TileMaps maps,
                                                             const __grid_constant__ Cameras cams,
                                                             const __grid_constant__ DecodeParams p, int nfr,
                                                             unsigned tiles_x, uint32_t* __restrict__ err) {
    constexpr int MPS = NPS ? NPS : MAX_PS;
    __shared__ float2 s_sc[MPS][HY][HX + 1];
    __shared__ float s_m[MPS][HY][HX + 1];
    const T* __restrict__ frames = static_cast<const T*>(cams.frames[blockIdx.y]);
    const int tid = threadIdx.x, n_ps = NPS ? NPS : p.n_ps;
    const int x0 = (int)(blockIdx.x % tiles_x) * TX, y0 = (int)(blockIdx.x / tiles_x) * TY;
    const size_t npx = (size_t)p.rows * p.cols;
    constexpr int XPAD = tma_xpad<T>(), BW = tma_bw<T>();
    extern __shared__ __align__(128) unsigned char box_raw[];  // [nfr][HY][BW] samples
    if constexpr (TMA) {
        __shared__ __align__(8) unsigned long long bar;
        const unsigned b = smem_addr(&bar);
        if (tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        if (tid == 0) {
            const unsigned bytes = (unsigned)(BW * HY * nfr * (int)sizeof(T));
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
            asm volatile(
                "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
                "[%5];" ::"r"(smem_addr(box_raw)),
                "l"(reinterpret_cast<unsigned long long>(&maps.m[blockIdx.y])), "r"(x0 - XPAD), "r"(y0 - 1), "r"(0), "r"(b)
                : "memory");
        }
        // bounded: a copy that never lands flags the error word; the tile waits
        // once more (bounded) for it before leaving
        if (!__syncthreads_and(mbar_wait0(b, TMA_POLLS))) {
            if (tid == 0) atomicOr(err, ERR_DECODE_COPY);
            mbar_wait0(b, TMA_POLLS);
            return;
        }
    }
    for (int h = tid; h < HX * HY; h += TX * TY) {
        const int hy = h / HX, hx = h - hy * HX;
        const int gy = min(max(y0 - 1 + hy, 0), p.rows - 1), gx = min(max(x0 - 1 + hx, 0), p.cols - 1);
        const T* box = reinterpret_cast<const T*>(box_raw) + (gy - (y0 - 1)) * BW + (gx - (x0 - XPAD));
        const T* pix = frames + (size_t)gy * p.cols + gx;
#pragma unroll
        for (int i = 0; i < MPS; i++) {
            if (i >= n_ps) break;
            const int f0 = NS ? i * NS : p.fbase[i];  // frequencies' frames are consecutive
            const int N = NS ? NS : p.shift[i];
            float2 sc = make_float2(0.f, 0.f);
            float m = 0.f;
            auto add = [&](int f, T v) {  // the S and C sums of one sample in one paired FMA
                sc = __ffma2_rn(make_float2(-p.sinv[f], p.cosv[f]), both((float)v), sc);
                m += (float)v;
            };
            if (TMA) {
#pragma unroll
                for (int k = 0; k < (NS ? NS : 32); k++) {  // 3..32 steps
                    if (k >= N) break;
                    add(f0 + k, box[(f0 + k) * (BW * HY)]);
                }
            } else if constexpr (NS > 0) {
                T v[NS];
#pragma unroll
                for (int k = 0; k < NS; k++) v[k] = __ldg(pix + (size_t)(f0 + k) * npx);
#pragma unroll
                for (int k = 0; k < NS; k++) add(f0 + k, v[k]);
            } else {
                int k = 0;
                for (; k + 4 <= N; k += 4) {  // four loads in flight
                    T v[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) v[u] = __ldg(pix + (size_t)(f0 + k + u) * npx);
#pragma unroll
                    for (int u = 0; u < 4; u++) add(f0 + k + u, v[u]);
                }
                for (; k < N; k++) add(f0 + k, __ldg(pix + (size_t)(f0 + k) * npx));
            }
            s_sc[i][hy][hx] = sc;
            s_m[i][hy][hx] = m;
        }
    }
    __syncthreads();
    const int tx = tid % TX, ty = tid / TX, x = x0 + tx, y = y0 + ty;
    if (x >= p.cols || y >= p.rows) return;
    const Outputs& out = cams.out[blockIdx.y];
    Pixel px;
    px.ok = true;
    px.mod = 0.f;
#pragma unroll
    for (int i = 0; i < MPS; i++) {
        if (i >= n_ps) break;
        float2 sc = make_float2(0.f, 0.f);
        float m = 0.f;
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) {
                const float w = p.w2d[a * 3 + b];
                sc = __ffma2_rn(both(w), s_sc[i][ty + a][tx + b], sc);
                m = fmaf(w, s_m[i][ty + a][tx + b], m);
            }
        take_frequency(p, i, sc.x, sc.y, m, out.mod != nullptr, px);
    }
    const size_t o = (size_t)y * p.cols + x;
    int g1 = 0, g2 = 0;
    if ((NPS == 1 || !NPS) && p.gray_bits > 0 && px.ok) {
        // codeword: bit set where N g > sum of the phase frames (exact in FP32)
        const float N = (float)p.shift[0], sum = s_m[0][ty + 1][tx + 1];
        auto bit = [&](int f) { return N * (float)__ldg(frames + (size_t)(p.gray_base + f) * npx + o) > sum ? 1 : 0; };
        int bin = 0;
        for (int f = 0; f < p.gray_bits; f++) {
            bin ^= bit(f);
            g1 = g1 << 1 | bin;
        }
        if (p.complementary) g2 = ((g1 << 1 | (bin ^ bit(p.gray_bits))) + 1) >> 1;
    }
    finish_pixel<MPS>(p, n_ps, px, g1, g2, o, out);
}

// cuTensorMapEncodeTiled from the driver, looked up once (no link to libcuda)
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    });
    return fn;
}

// The cameras' tensor maps, or false where the copy does not apply (row pitch or base
// not 16-byte aligned, too many frames, an image smaller than the box).
template <typename T>
bool tile_maps(const Cameras& cams, int n, const DecodeParams& p, int nfr, TileMaps& maps) {
    const size_t pitch = (size_t)p.cols * sizeof(T);
    if (nfr > TMA_MAX_FRAMES || pitch % 16 != 0 || p.cols < tma_bw<T>() || p.rows < HY) return false;
    for (int c = 0; c < n; c++)
        if (((uintptr_t)cams.frames[c] & 15) != 0) return false;
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)p.cols, (cuuint64_t)p.rows, (cuuint64_t)nfr};
    const cuuint64_t strides[2] = {(cuuint64_t)pitch, (cuuint64_t)pitch * p.rows};
    const cuuint32_t box[3] = {(cuuint32_t)tma_bw<T>(), (cuuint32_t)HY, (cuuint32_t)nfr};
    const cuuint32_t one[3] = {1, 1, 1};
    for (int c = 0; c < n; c++)
        if (enc(&maps.m[c], sizeof(T) == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 3,
                const_cast<void*>(cams.frames[c]), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    return true;
}

// HDR fit of one frequency at a pixel pair (JSLAB_HDRPhaseFit.h:10-61 and
// JSLAB_PhaseShiftDecoder_V2.cpp:73-90): raw samples with 0 <= I < saturation
// enter an equal-variance least-squares fit of I = A + C cos d - S sin d
// (solved here from the 3x3 normal equations, the reference's cached
// pseudo-inverse of the same subset); fewer than three samples, amplitude
// hypot(C, S) <= min_amp or A <= 1e-3 reject the pixel.  Returns the sums the
// phase-shift path would have formed: S N/2, C N/2, A N.  A sample's mask is the
// factor 1 or 0 of its terms (exact), so both pixels run as one.
template <typename T, int NS>
__device__ __forceinline__ void hdr_fit(const T* q, size_t npx, bool pair, int d, const DecodeParams& p, int i, float2& S,
                                        float2& C, float2& M, bool& ok0, bool& ok1) {
    const float2 zero = both(0.f);
    auto below = [](float v, float limit) {  // 1 or 0
        float r;
        asm("set.lt.f32.f32 %0, %1, %2;" : "=f"(r) : "f"(v), "f"(limit));
        return r;
    };
    float2 m00 = zero, m01 = zero, m02 = zero, m11 = zero, m12 = zero, m22 = zero, r0 = zero, r1 = zero, r2 = zero;
    const int N = NS ? NS : p.shift[i], f0 = NS ? i * NS : p.fbase[i];
    auto add = [&](int f, unsigned w) {
        float2 v = unpack<T>(w);
        const float2 in = make_float2(below(v.x, p.hdr_sat), below(v.y, p.hdr_sat));
        const float2 c = make_float2(in.x * p.cosv[f], in.y * p.cosv[f]);
        const float2 s = make_float2(in.x * -p.sinv[f], in.y * -p.sinv[f]);
        v = __fmul2_rn(in, v);
        m00 = __fadd2_rn(m00, in);
        m01 = __fadd2_rn(m01, c);
        m02 = __fadd2_rn(m02, s);
        m11 = __ffma2_rn(c, c, m11);
        m12 = __ffma2_rn(c, s, m12);
        m22 = __ffma2_rn(s, s, m22);
        r0 = __fadd2_rn(r0, v);
        r1 = __ffma2_rn(c, v, r1);
        r2 = __ffma2_rn(s, v, r2);
    };
    if constexpr (NS > 0) {
        unsigned w[NS];
        load_pairs(q + (size_t)f0 * npx, npx, pair, d, w);
#pragma unroll
        for (int k = 0; k < NS; k++) add(f0 + k, w[k]);
    } else {
        int k = 0;
        for (; k + 4 <= N; k += 4) {  // four loads in flight
            unsigned w[4];
            load_pairs(q + (size_t)(f0 + k) * npx, npx, pair, d, w);
#pragma unroll
            for (int u = 0; u < 4; u++) add(f0 + k + u, w[u]);
        }
        for (; k < N; k++) {
            unsigned w[1];
            load_pairs(q + (size_t)(f0 + k) * npx, npx, pair, d, w);
            add(f0 + k, w[0]);
        }
    }
    auto neg = [](float2 a) { return make_float2(-a.x, -a.y); };
    // symmetric 3x3 inverse by cofactors
    const float2 c00 = __ffma2_rn(m11, m22, __fmul2_rn(neg(m12), m12));
    const float2 c01 = __ffma2_rn(m02, m12, __fmul2_rn(neg(m01), m22));
    const float2 c02 = __ffma2_rn(m01, m12, __fmul2_rn(neg(m02), m11));
    const float2 det = __ffma2_rn(m00, c00, __ffma2_rn(m01, c01, __fmul2_rn(m02, c02)));
    const float2 c11 = __ffma2_rn(m00, m22, __fmul2_rn(neg(m02), m02));
    const float2 c12 = __ffma2_rn(m01, m02, __fmul2_rn(neg(m00), m12));
    const float2 c22 = __ffma2_rn(m00, m11, __fmul2_rn(neg(m01), m01));
    const float2 id = make_float2(__frcp_rn(det.x), __frcp_rn(det.y));
    const float2 A = __fmul2_rn(__ffma2_rn(c00, r0, __ffma2_rn(c01, r1, __fmul2_rn(c02, r2))), id);
    C = __fmul2_rn(__ffma2_rn(c01, r0, __ffma2_rn(c11, r1, __fmul2_rn(c12, r2))), id);
    S = __fmul2_rn(__ffma2_rn(c02, r0, __ffma2_rn(c12, r1, __fmul2_rn(c22, r2))), id);
    auto accept = [&](float n, float det, float A, float C, float S) {
        if (n < 3.f || !(fabsf(det) > 1e-6f * n * n * n) || !(A > 1e-3f)) return false;
        // hypot(C, S) > min_amp, by squares where those decide beyond rounding
        const float q = fmaf(C, C, S * S), t = p.hdr_min_amp * p.hdr_min_amp;
        if (q > 1.00001f * t) return true;
        if (q < 0.99999f * t) return false;
        return hypotf(C, S) > p.hdr_min_amp;
    };
    ok0 = accept(m00.x, det.x, A.x, C.x, S.x);
    ok1 = accept(m00.y, det.y, A.y, C.y, S.y);
    const float2 n2 = both((float)N), half = both(0.5f);
    S = __fmul2_rn(__fmul2_rn(S, n2), half);
    C = __fmul2_rn(__fmul2_rn(C, n2), half);
    M = __fmul2_rn(A, n2);
}

// HDR decode: raw samples, no pre-blur (saturation is classified before any
// blur), a pixel pair per thread.  Bound by instruction issue (nine sums per
// sample): paired over two pixels and without branches 35 us for 24 frames of
// 1280x1024, 64 us one pixel at a time.  Step counts without code of their own load
// four samples at a time: 12 steps, 16-bit, 2448x2048 318 us one by one, 176 so.
template <typename T, int NPS, int NS>
__global__ void __launch_bounds__(128) decode_hdr_kernel(const __grid_constant__ Cameras cams,
                                                         const __grid_constant__ DecodeParams p, int aligned_cams) {
    const T* __restrict__ frames = static_cast<const T*>(cams.frames[blockIdx.y]);
    const Outputs& out = cams.out[blockIdx.y];
    const int aligned = aligned_cams >> blockIdx.y & 1;
    const int half = (p.cols + 1) / 2;
    const size_t t = (size_t)blockIdx.x * 128 + threadIdx.x;
    const int y = (int)(t / (unsigned)half);
    if (y >= p.rows) return;
    const int x = 2 * (int)(t - (size_t)y * half);
    const size_t npx = (size_t)p.rows * p.cols;
    const int n_ps = NPS < MAX_PS ? NPS : p.n_ps;
    const T* q = frames + (size_t)y * p.cols + x;
    const int d = x + 1 < p.cols ? 1 : 0;
    Pixel p0, p1;
    p0.ok = p1.ok = true;
#pragma unroll
    for (int i = 0; i < NPS; i++) {
        if (i >= n_ps) break;
        float2 S, C, M;
        bool f0, f1;
        hdr_fit<T, NS>(q, npx, aligned, d, p, i, S, C, M, f0, f1);
        p0.ok = p0.ok && f0;
        p1.ok = p1.ok && f1;
        take_frequency(p, i, S.x, C.x, M.x, out.mod != nullptr, p0);
        take_frequency(p, i, S.y, C.y, M.y, out.mod != nullptr, p1);
    }
    const size_t o = (size_t)y * p.cols + x;
    finish_pixel<NPS>(p, n_ps, p0, 0, 0, o, out);
    if (d) finish_pixel<NPS>(p, n_ps, p1, 0, 0, o + 1, out);
}

// Strips or tiles, where both have the step count (tma: the tiles come by bulk copy;
// n cameras).  Strips issue least, but a row at a time: they win once the launch is
// many waves deep.  us, tiles / strips: three frequencies of four steps, 8-bit,
// hierarchical, 1280x1024 23 / 24, 1626x1236 36 / 34, 2448x2048 83 / 74; heterodyne 26 /
// 28, 40 / 41, 92 / 91; both cameras of 1280x1024 even, of 2448x2048 20 less in strips.
// Eight steps, bulk copy, 8-bit 2448x2048: 108 / 115 (4096x3000: 258 / 261), 16-bit 112 /
// 111 (267 / 252); without it (2501x2092) 139 / 118 and 168 / 114, 16-bit from 487x365
// (8.2 / 8.2) on.  Other step counts hold too few samples ahead in a strip (five steps,
// 8-bit, 2448x2048: 127 / 304), Gray codes read their frames late (four steps, five
// bits: 2448x2048 76 / 91, 1626x1236 28 / 29), and small images wait a strip's rows
// out (three by eight steps, 64x64: 3.5 / 6).
template <typename T>
bool use_strips(const DecodeParams& p, int n, int ns, bool tma) {
    if (p.n_ps != 3 || (ns != 4 && ns != 8)) return false;
    const double px = (double)n * p.rows * p.cols;
    if (ns == 8 && tma && sizeof(T) == 1) return false;
    return px >= (ns == 8 && !tma && sizeof(T) == 2 ? 0.18e6 : 1.5e6);
}

template <typename T>
void launch_decode(zim_ctx* ctx, const Cameras& cams, int n, const DecodeParams& p, cudaStream_t st) {
    int aligned = 0;  // bit per camera
    for (int c = 0; c < n; c++)
        aligned |= (p.cols % 2 == 0 && ((uintptr_t)cams.frames[c] & (2 * sizeof(T) - 1)) == 0) << c;
    int ns = p.shift[0];
    for (int i = 1; i < p.n_ps; i++) ns = p.shift[i] == ns ? ns : 0;
    if (p.hdr) {
        const unsigned blocks = (unsigned)(((size_t)p.rows * ((p.cols + 1) / 2) + 127) / 128);
        auto k = p.n_ps == 3 && ns == 8 ? decode_hdr_kernel<T, 3, 8>
                 : p.n_ps == 3 && ns == 4 ? decode_hdr_kernel<T, 3, 4> : decode_hdr_kernel<T, MAX_PS, 0>;
        k<<<dim3(blocks, n), 128, 0, st>>>(cams, p, aligned);
        ctx->launches += 1;
        return;
    }
    int nfr = 0;
    for (int i = 0; i < p.n_ps; i++) nfr += p.shift[i];
    TileMaps maps{};
    const bool tma = tile_maps<T>(cams, n, p, nfr, maps);
    auto by_steps = [&](auto run) {  // the step counts with code of their own
        constexpr std::integral_constant<int, 0> c0;
        constexpr std::integral_constant<int, 1> c1;
        constexpr std::integral_constant<int, 3> c3;
        constexpr std::integral_constant<int, 4> c4;
        constexpr std::integral_constant<int, 8> c8;
        if (p.n_ps == 3 && ns == 4) run(c3, c4);
        else if (p.n_ps == 3 && ns == 8) run(c3, c8);
        else if (p.n_ps == 1 && ns == 4) run(c1, c4);
        else run(c0, c0);
    };
    const bool strips = use_strips<T>(p, n, ns, tma);
    by_steps([&](auto nps, auto nsteps) {
        constexpr int NPS = decltype(nps)::value, NS = decltype(nsteps)::value;
        if constexpr (NPS == 3) {
            if (strips) {
                const int nstrips = (p.cols + STRIP - 1) / STRIP;
                const int band = strip_band(ctx, nstrips * n, p.rows, DEC_MIN_WARPS);
                const long long warps = (long long)nstrips * ((p.rows + band - 1) / band);
                const dim3 blocks((unsigned)((warps + DEC_WARPS - 1) / DEC_WARPS), n);
                if (n == 2)
                    decode_strips_kernel<T, NPS, NS><<<blocks, 32 * DEC_WARPS, 0, st>>>(cams, p, band, nstrips);
                else
                    decode_strip_kernel<T, NPS, NS><<<blocks, 32 * DEC_WARPS, 0, st>>>(
                        static_cast<const T*>(cams.frames[0]), p, band, nstrips, cams.out[0]);
                return;
            }
        }
        const unsigned tiles_x = (p.cols + TX - 1) / TX;
        const dim3 grid(tiles_x * (unsigned)((p.rows + TY - 1) / TY), n);
        if (tma)
            decode_tile_kernel<T, NPS, NS, true><<<grid, TX * TY, sizeof(T) * tma_bw<T>() * HY * nfr, st>>>(
                maps, cams, p, nfr, tiles_x, ctx->d_error);
        else
            decode_tile_kernel<T, NPS, NS, false><<<grid, TX * TY, 0, st>>>(maps, cams, p, nfr, tiles_x, ctx->d_error);
    });
    ctx->launches += 1;
}

// Absolute phase as f64 (startCalculate's CV_64F map; 0 where invalid), with
// the optional 3x3 post-smooth (fixed [1/4 1/2 1/4] kernel, BORDER_REPLICATE):
// post_smooth 1 blurs the phase map as is; 2 is the HDR form, the blur divided
// by the blurred validity, 0 at invalid pixels (JSLAB_PhaseShiftDecoder_V2.cpp:280-291);
// 3 is an HDR decode without smoothing.  An HDR decode marks invalid pixels
// with order -1 (a plain decode zeroes them, and Gray code can give a valid -1).
__global__ void phase_f64_kernel(const int32_t* __restrict__ order, const float* __restrict__ res, int rows, int cols,
                                 int post_smooth, double* __restrict__ out) {
    int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= cols || y >= rows) return;
    const size_t oc = (size_t)y * cols + x;
    const bool hdr = post_smooth >= 2;
    if (post_smooth == 0 || post_smooth == 3) {
        out[oc] = hdr && order[oc] < 0 ? 0.0 : 6.283185307179586 * order[oc] + (double)res[oc];
        return;
    }
    if (hdr && order[oc] < 0) {
        out[oc] = 0.0;
        return;
    }
    double P = 0, W = 0;
    for (int a = -1; a <= 1; a++) {
        int yy = min(max(y + a, 0), rows - 1);
        for (int b = -1; b <= 1; b++) {
            int xx = min(max(x + b, 0), cols - 1);
            int w = (a == 0 ? 2 : 1) * (b == 0 ? 2 : 1);
            size_t o = (size_t)yy * cols + xx;
            if (hdr && order[o] < 0) continue;
            P += w * (6.283185307179586 * order[o] + (double)res[o]);
            W += w;
        }
    }
    out[oc] = hdr ? P / W : P / 16.0;
}

}  // namespace

void zim_decode_params_launch(zim_ctx* ctx, int n, const void* const* frames, int sample_type,
                              const zt::DecodeParams& p, int32_t* const* order, float* const* residual, float* mod,
                              uint8_t* valid, cudaStream_t st) {
    Cameras cams{};
    for (int c = 0; c < n; c++) {
        cams.frames[c] = frames[c];
        cams.out[c] = Outputs{order[c], residual[c], mod, valid};
    }
    if (sample_type == ZIM_SAMPLE_U8) launch_decode<uint8_t>(ctx, cams, n, p, st);
    else launch_decode<uint16_t>(ctx, cams, n, p, st);
}

zim_status zim_decode_launch(zim_ctx* ctx, const zim_decode_config* cfg, int n, const void* const* frames,
                             int sample_type, int rows, int cols, int32_t* const* order, float* const* residual,
                             float* mod, uint8_t* valid, cudaStream_t st) {
    DecodeParams p;
    zt::decode_params(cfg, rows, cols, p);
    zim_decode_params_launch(ctx, n, frames, sample_type, p, order, residual, mod, valid, st);
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}

extern "C" ZIM_API zim_status zim_decode(zim_ctx* ctx, const zim_decode_config* cfg, const void* frames,
                                         int sample_type, int rows, int cols, int32_t* order, float* residual,
                                         float* mod, uint8_t* valid, void* stream) {
    if (!ctx) return ZIM_ERR_INVALID_ARG;
    zim_status s = zim_decode_validate(cfg);
    if (s != ZIM_OK) return zim_fail(ctx, s, "invalid decode config");
    if (!frames || !order || !residual) return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "null argument");
    if (rows <= 0 || cols <= 0 || (size_t)rows * cols > ((size_t)1 << 31))
        return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "bad image size %dx%d", cols, rows);
    if (sample_type != ZIM_SAMPLE_U8 && sample_type != ZIM_SAMPLE_U16)
        return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "bad sample type");
    ZIM_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return zim_decode_launch(ctx, cfg, 1, &frames, sample_type, rows, cols, &order, &residual, mod, valid,
                             zim_stream(stream));
}

extern "C" ZIM_API zim_status zim_decode_phase_f64(zim_ctx* ctx, const int32_t* order, const float* residual, int rows,
                                                   int cols, int post_smooth, double* phase, void* stream) {
    if (!ctx) return ZIM_ERR_INVALID_ARG;
    if (!order || !residual || !phase || rows <= 0 || cols <= 0)
        return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "bad argument");
    ZIM_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    dim3 blk(256), grd((cols + 255) / 256, rows);
    phase_f64_kernel<<<grd, blk, 0, zim_stream(stream)>>>(order, residual, rows, cols, post_smooth, phase);
    ctx->launches += 1;
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}
