// recon.cu -- disparity median + Q reprojection, the reference's pixel-window
// point-cloud filters (3x3 Gaussian, radius outlier) and PointXYZ compaction.
//
// Reference: PhaseShiftGrayCode3D/src/JSLAB_PhaseEpipolarReconstructor_V2.cpp
//   medianBlur(5) :405-410, reprojection :414-461, Gaussian :79-124, ROR :126-195;
//   GPU port JSLAB_PhaseEpipolarReconstructor_V2_GPU.cu:119-347.
#include <cmath>

#include "zim_tiles.cuh"

namespace {

using zt::ReprojParams;
using zt::RX;
using zt::RY;

__global__ void __launch_bounds__(32 * zt::MED_WARPS, 3) median_reproject_kernel(
    const float* __restrict__ disp, int rows, int cols, const __grid_constant__ ReprojParams p, int band, int nstrips,
    float* __restrict__ disp_out, float* __restrict__ xyz, uint8_t* __restrict__ mask) {
    __shared__ zt::MedianSmem sm;
    const int w = threadIdx.x >> 5, id = blockIdx.x * zt::MED_WARPS + w;
    const int y0 = (id / nstrips) * band;
    if (y0 < rows)
        zt::median_reproject_strip(disp, rows, cols, p, id % nstrips, y0, min(y0 + band, rows), w, sm, disp_out, xyz,
                                   mask);
}

constexpr int PXG_WARPS = 4;
constexpr size_t ROR_SMEM = 52 * 1024;  // shared memory of a radius-filter tile taller than RY rows
// Rows of a radius-filter tile: tall tiles stage less halo per point, but few of them
// end in a nearly empty wave.  us, with this rule / with 32 rows throughout: 11 x 11,
// nobody with enough neighbours, 1024 x 768 46.5 / 51.7; 21 x 21 155 / 197; the
// default filter 1280 x 1024 30.2 / 35.8.
inline int ror_rows(int sms, int rows, int cols, int hw) {
    int th = 32;
    auto blocks = [&](int th) { return (long long)((cols + RX - 1) / RX) * ((rows + th - 1) / th); };
    while (th > RY && (zt::ror_smem_bytes(hw, th) > ROR_SMEM || blocks(th) < (th == 32 ? 64ll : 12ll) * sms)) th /= 2;
    return th;
}
__global__ void __launch_bounds__(32 * PXG_WARPS) px_gaussian_kernel(const float* __restrict__ xyz,
                                                                     const uint8_t* __restrict__ mask, int rows,
                                                                     int cols, int band, int nstrips, float w00,
                                                                     float w01, float w11, float* __restrict__ out,
                                                                     uint8_t* __restrict__ mask_out) {
    const int id = blockIdx.x * PXG_WARPS + (threadIdx.x >> 5), y0 = (id / nstrips) * band;
    if (y0 < rows)
        zt::px_gaussian_strip(xyz, mask, rows, cols, id % nstrips, y0, min(y0 + band, rows), w00, w01, w11, out,
                              mask_out);
}

template <bool WIDE>
__global__ void __launch_bounds__(RX* RY) ror_kernel(const float* __restrict__ xyz, const uint8_t* __restrict__ mask,
                                                     int rows, int cols, int th, float r2, int min_nb, int hw,
                                                     float* __restrict__ out, uint8_t* __restrict__ mask_out) {
    extern __shared__ float4 ror_smem[];
    zt::ror_tile<WIDE>(xyz, mask, rows, cols, blockIdx.x * RX, blockIdx.y * th, th, threadIdx.x, r2, min_nb, hw, ror_smem, out,
                 mask_out);
}

constexpr int CB = 1024;  // compaction block

__global__ void compact_count_kernel(const uint8_t* __restrict__ mask, size_t n, uint32_t* __restrict__ counts) {
    __shared__ uint32_t warp_sums[CB / 32];
    size_t i = (size_t)blockIdx.x * CB + threadIdx.x;
    uint32_t v = (i < n && mask[i]) ? 1u : 0u;
    uint32_t b = __ballot_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = __popc(b);
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t s = warp_sums[threadIdx.x];
        for (int off = 16; off; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
        if (threadIdx.x == 0) counts[blockIdx.x] = s;
    }
}

// Single-CTA exclusive scan of the block counts; total goes to count_dev.
__global__ void compact_scan_kernel(uint32_t* __restrict__ counts, int nb, uint64_t* __restrict__ count_dev) {
    __shared__ uint32_t carry_s;
    __shared__ uint32_t wsum[32];
    if (threadIdx.x == 0) carry_s = 0;
    __syncthreads();
    for (int base = 0; base < nb; base += 1024) {
        int i = base + threadIdx.x;
        uint32_t v = i < nb ? counts[i] : 0;
        uint32_t x = v;
        int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, x, off);
            if (lane >= off) x += t;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        if (w == 0) {
            uint32_t s = wsum[lane];
            for (int off = 1; off < 32; off <<= 1) {
                uint32_t t = __shfl_up_sync(0xffffffffu, s, off);
                if (lane >= off) s += t;
            }
            wsum[lane] = s;
        }
        __syncthreads();
        uint32_t incl = x + (w > 0 ? wsum[w - 1] : 0);
        uint32_t carry = carry_s;
        if (i < nb) counts[i] = carry + incl - v;
        __syncthreads();
        if (threadIdx.x == 1023) carry_s = carry + incl;
        __syncthreads();
    }
    if (threadIdx.x == 0) *count_dev = carry_s;
}

// Record layouts the compaction can emit for each valid point, in row order.
enum Emit { EMIT_POINTXYZ, EMIT_PLY_XYZ, EMIT_PLY_XYZ_GRAY };

// Binary little-endian PLY vertex bodies (savePointCloudToPlyBinary and
// savePointCloudToPlyBinaryWithGray, main.cpp:85-160): float x, y, z, then for
// the grey variant the grey value three times as uchar red, green, blue.
template <int E>
__device__ __forceinline__ void emit(const float* __restrict__ xyz, const uint8_t* __restrict__ gray, size_t i,
                                     uint32_t pos, void* __restrict__ out) {
    const float x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
    if (E == EMIT_POINTXYZ) {
        zim_point_xyz p;
        p.x = x; p.y = y; p.z = z;
        p.pad = 1.0f;
        static_cast<zim_point_xyz*>(out)[pos] = p;
    } else if (E == EMIT_PLY_XYZ) {
        float* r = static_cast<float*>(out) + 3 * (size_t)pos;
        r[0] = x; r[1] = y; r[2] = z;
    } else {
        uint8_t* r = static_cast<uint8_t*>(out) + 15 * (size_t)pos;  // byte-aligned records
        const float v[3] = {x, y, z};
        const uint8_t* b = reinterpret_cast<const uint8_t*>(v);
#pragma unroll
        for (int k = 0; k < 12; k++) r[k] = b[k];
        const uint8_t g = gray ? gray[i] : (uint8_t)255;
        r[12] = g; r[13] = g; r[14] = g;
    }
}

template <int E>
__global__ void compact_write_kernel(const float* __restrict__ xyz, const uint8_t* __restrict__ mask, size_t n,
                                     const uint32_t* __restrict__ offsets, const uint8_t* __restrict__ gray,
                                     void* __restrict__ out) {
    __shared__ uint32_t warp_off[CB / 32];
    size_t i = (size_t)blockIdx.x * CB + threadIdx.x;
    bool v = i < n && mask[i];
    uint32_t b = __ballot_sync(0xffffffffu, v);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) warp_off[w] = __popc(b);
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t s = warp_off[threadIdx.x], x = s;
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, x, off);
            if (threadIdx.x >= off) x += t;
        }
        warp_off[threadIdx.x] = x - s;
    }
    __syncthreads();
    if (v) emit<E>(xyz, gray, i, offsets[blockIdx.x] + warp_off[w] + __popc(b & ((1u << lane) - 1u)), out);
}

}  // namespace

zim_status zim_median_reproject_launch(zim_ctx* ctx, const zim_recon_config* cfg, const float* disp, int rows,
                                       int cols, float* disp_out, float* xyz, uint8_t* mask, cudaStream_t st) {
    ReprojParams p;
    zt::reproj_params(ctx->Q, ctx->R1, cfg, p);
    for (int k = 0; k < 3; k++) p.poly[k] = ctx->d_poly[k];
    zim_median_strips(ctx, p, disp, rows, cols, disp_out, xyz, mask, st);
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}

void zim_median_strips(zim_ctx* ctx, const ReprojParams& p, const float* disp, int rows, int cols, float* disp_out,
                       float* xyz, uint8_t* mask, cudaStream_t st) {
    const int nstrips = (cols + zt::MSTRIP - 1) / zt::MSTRIP;
    const int band = strip_band(ctx, nstrips, rows, 32);
    const long long warps = (long long)nstrips * ((rows + band - 1) / band);
    median_reproject_kernel<<<(unsigned)((warps + zt::MED_WARPS - 1) / zt::MED_WARPS), 32 * zt::MED_WARPS, 0, st>>>(
        disp, rows, cols, p, band, nstrips, disp_out, xyz, mask);
    ctx->launches += 1;
}

zim_status zim_px_gaussian_launch(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows, int cols, float* out,
                                  uint8_t* mask_out, cudaStream_t st) {
    float w00, w01, w11;
    zt::px_gaussian_weights(w00, w01, w11);
    const int nstrips = (cols + zt::PXG_STRIP - 1) / zt::PXG_STRIP, band = strip_band(ctx, nstrips, rows, 32);
    const long long warps = (long long)nstrips * ((rows + band - 1) / band);
    px_gaussian_kernel<<<(unsigned)((warps + PXG_WARPS - 1) / PXG_WARPS), 32 * PXG_WARPS, 0, st>>>(
        xyz, mask, rows, cols, band, nstrips, w00, w01, w11, out, mask_out);
    ctx->launches += 1;
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}

zim_status zim_ror_launch(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows, int cols, float radius,
                          int min_neighbors, int window_size, float* out, uint8_t* mask_out, cudaStream_t st) {
    const int hw = window_size / 2;
    const int th = ror_rows(ctx->sm_count > 0 ? ctx->sm_count : 152, rows, cols, hw);
    const size_t smem = zt::ror_smem_bytes(hw, th);
    auto kern = zt::ror_wide(hw, radius) ? ror_kernel<true> : ror_kernel<false>;
    ZIM_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grd((cols + RX - 1) / RX, (rows + th - 1) / th);
    kern<<<grd, RX * RY, smem, st>>>(xyz, mask, rows, cols, th, radius * radius, min_neighbors, hw, out, mask_out);
    ctx->launches += 1;
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}

zim_status zim_compact_launch(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows, int cols,
                              zim_point_xyz* points, uint64_t* count_dev, cudaStream_t st) {
    size_t n = (size_t)rows * cols;
    int nb = (int)((n + CB - 1) / CB);
    uint32_t* counts = (uint32_t*)zim_scratch_take(ctx, (size_t)nb * 4);
    if (!counts) return zim_fail(ctx, ZIM_ERR_OUT_OF_MEMORY, "compaction scratch");
    compact_count_kernel<<<nb, CB, 0, st>>>(mask, n, counts);
    compact_scan_kernel<<<1, 1024, 0, st>>>(counts, nb, count_dev);
    compact_write_kernel<EMIT_POINTXYZ><<<nb, CB, 0, st>>>(xyz, mask, n, counts, nullptr, points);
    ctx->launches += 3;
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}

static zim_status pack_ply_launch(zim_ctx* ctx, const float* xyz, const uint8_t* mask, const uint8_t* gray,
                                  int with_gray, int rows, int cols, void* records, uint64_t* count_dev,
                                  cudaStream_t st) {
    size_t n = (size_t)rows * cols;
    int nb = (int)((n + CB - 1) / CB);
    uint32_t* counts = (uint32_t*)zim_scratch_take(ctx, (size_t)nb * 4);
    if (!counts) return zim_fail(ctx, ZIM_ERR_OUT_OF_MEMORY, "compaction scratch");
    compact_count_kernel<<<nb, CB, 0, st>>>(mask, n, counts);
    compact_scan_kernel<<<1, 1024, 0, st>>>(counts, nb, count_dev);
    if (with_gray)
        compact_write_kernel<EMIT_PLY_XYZ_GRAY><<<nb, CB, 0, st>>>(xyz, mask, n, counts, gray, records);
    else
        compact_write_kernel<EMIT_PLY_XYZ><<<nb, CB, 0, st>>>(xyz, mask, n, counts, nullptr, records);
    ctx->launches += 3;
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}

zim_ray_model zim_rays_of(const zim_ctx* ctx, bool rectified_coords, int ox, int oy) {
    if (!ctx->calibrated) return zim_ray_model{};
    return zim_rays_from(ctx->Q, ctx->R1, rectified_coords, ox, oy);
}

zim_ray_model zim_rays_from(const double* Q, const double* R1, bool rectified_coords, int ox, int oy) {
    zim_ray_model r;
    if (!(Q[11] != 0.0)) return r;
    // Q reprojects pixel (u, v) along (u + Q03, v + Q13, Q23)
    r.cx = (float)-Q[3];
    r.cy = (float)-Q[7];
    r.f = (float)Q[11];
    if (!rectified_coords)
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) r.R[3 * a + b] = (float)R1[3 * b + a];  // R1^T
    r.ox = ox;
    r.oy = oy;
    r.valid = 1;
    return r;
}

zim_status zim_check_reproject(zim_ctx* ctx, const zim_recon_config* cfg) {
    if (cfg->reproject_model != 0 && cfg->reproject_model != 1)
        return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "reproject_model must be 0 (Q) or 1 (polynomial maps)");
    // startCalculate_v2 writes no point without V2 coefficients (V2.cpp:505-548)
    if (cfg->reproject_model == 1 && !ctx->d_poly[0])
        return zim_fail(ctx, ZIM_ERR_NOT_CALIBRATED, "reproject_model 1 needs zim_set_poly_calib");
    return ZIM_OK;
}

static zim_status check_cloud(zim_ctx* ctx, const void* a, const void* b, const void* c, int rows, int cols) {
    if (!ctx) return ZIM_ERR_INVALID_ARG;
    if (!a || !b || !c) return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "null argument");
    if (rows <= 0 || cols <= 0) return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "bad size");
    ZIM_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return ZIM_OK;
}

extern "C" ZIM_API zim_status zim_median_reproject(zim_ctx* ctx, const zim_recon_config* cfg, const float* disp,
                                                   int rows, int cols, float* disp_out, float* xyz, uint8_t* mask,
                                                   void* stream) {
    zim_status s = check_cloud(ctx, disp, xyz, mask, rows, cols);
    if (s) return s;
    if (!cfg) return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "null config");
    if (!ctx->calibrated) return zim_fail(ctx, ZIM_ERR_NOT_CALIBRATED, "not calibrated");
    s = zim_check_reproject(ctx, cfg);
    if (s) return s;
    if (cfg->reproject_model == 1 && (rows != ctx->poly_h || cols != ctx->poly_w))
        return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "disparity %dx%d differs from the coefficient maps %dx%d", cols, rows,
                        ctx->poly_w, ctx->poly_h);
    return zim_median_reproject_launch(ctx, cfg, disp, rows, cols, disp_out, xyz, mask, zim_stream(stream));
}

extern "C" ZIM_API zim_status zim_filter_px_gaussian(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows,
                                                     int cols, float* out, uint8_t* mask_out, void* stream) {
    zim_status s = check_cloud(ctx, xyz, mask, out, rows, cols);
    if (s) return s;
    return zim_px_gaussian_launch(ctx, xyz, mask, rows, cols, out, mask_out, zim_stream(stream));
}

extern "C" ZIM_API zim_status zim_filter_ror(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows, int cols,
                                             float radius, int min_neighbors, int window_size, float* out,
                                             uint8_t* mask_out, void* stream) {
    zim_status s = check_cloud(ctx, xyz, mask, out, rows, cols);
    if (s) return s;
    if (!mask_out || window_size < 0 || window_size > ZIM_MAX_ROR_WINDOW || min_neighbors < 0)
        return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "bad ROR argument");
    return zim_ror_launch(ctx, xyz, mask, rows, cols, radius, min_neighbors, window_size, out, mask_out,
                          zim_stream(stream));
}

extern "C" ZIM_API zim_status zim_compact_points(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows,
                                                 int cols, zim_point_xyz* points, uint64_t* count_dev, void* stream) {
    zim_status s = check_cloud(ctx, xyz, mask, points, rows, cols);
    if (s) return s;
    if (!count_dev) return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "null count");
    size_t nb = ((size_t)rows * cols + CB - 1) / CB;
    s = zim_scratch_reserve(ctx, nb * 4 + 256);
    if (s) return s;
    zim_scratch_reset(ctx);
    return zim_compact_launch(ctx, xyz, mask, rows, cols, points, count_dev, zim_stream(stream));
}

extern "C" ZIM_API zim_status zim_pack_ply(zim_ctx* ctx, const float* xyz, const uint8_t* mask, const uint8_t* gray,
                                           int with_gray, int rows, int cols, void* records, uint64_t* count_dev,
                                           void* stream) {
    zim_status s = check_cloud(ctx, xyz, mask, records, rows, cols);
    if (s) return s;
    if (!count_dev) return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "null count");
    size_t nb = ((size_t)rows * cols + CB - 1) / CB;
    s = zim_scratch_reserve(ctx, nb * 4 + 256);
    if (s) return s;
    zim_scratch_reset(ctx);
    return pack_ply_launch(ctx, xyz, mask, gray, with_gray, rows, cols, records, count_dev, zim_stream(stream));
}
