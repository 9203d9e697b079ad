// grid.cu -- whole-cloud filters of an organised cloud: the PCL-style
// StatisticalOutlierRemoval (exact k nearest neighbours) and the metric
// (millimetre-sigma) Gaussian.
//
// Neither filter exists in the reference tree (PCL is linked but never
// included, PhaseShiftGrayCode3D/PCL114_Release_x64.props:17-18); SOR follows
// PCL's documented StatisticalOutlierRemoval algorithm: mean distance to the k
// nearest neighbours, threshold mean + std_mul * stddev, keep d <= threshold.
//
// Both run a window pass over the pixels around each point first and leave the
// few points it cannot settle to the cloud's bounding-box tree (zim_leaf.cuh).
//
// SOR on a cloud with pixel rays (the organised cloud of the calibrated size):
//   window pass: one thread per pixel walks its 15x15 window in a spiral with
//            the k + 1 nearest in groups of five, certified exact by a bound on
//            the distance to every point seen along another pixel's ray;
//   tree search: one warp per remaining point reads the leaves whose box lies
//            within the (k + 1)-th distance held.
// Without pixel rays a tile search takes the window pass's place: a uniform
// grid with cells of a few pixel spacings (a hash table of (offset, count)
// pairs), one CTA per 16x8 pixel tile gathering the points of the tile's cell
// box (dilated by TILE_DILATE cells) into shared memory; every thread scans the
// same candidate list and is exact once it holds k + 1 candidates within its
// distance to the box boundary.  A visited point's cell is re-derived from its
// coordinates, so hash collisions never count a point twice.  Every path sums
// the same k + 1 roots in fixed point, so a query's mean distance has the same
// bits whichever path settles it.
//
// The metric Gaussian: a window pass with the same ray bound; the queries it
// cannot certify (all of them without pixel rays) are summed over the tree's
// leaves in 64-bit fixed point.  The SOR statistics are summed in a fixed
// order: both filters are deterministic.

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <utility>

#include "zim_leaf.cuh"

namespace {

constexpr int GB = 256;          // threads for pixel-parallel kernels
constexpr int KNN_MAX_K1 = 64;   // k + 1 <= 64
constexpr int SCAN_B = 1024;
constexpr int FINE_RINGS = 2;    // tile search's fallback rings of cells
constexpr int TS_WARPS = 4;      // tree search: warps per CTA
// md marker of a deferred query whose bound on the (k + 1)-th squared distance
// is handed on in the bound array (md = -1: no bound)
constexpr float MD_BOUND = -3.f;
constexpr int TILE_X = 16, TILE_Y = 8, TILE_T = TILE_X * TILE_Y;
// the window passes' tiles: taller tiles stage less halo per query
constexpr int WT_X = 16, WT_Y = 16, WT_T = WT_X * WT_Y;
constexpr int TILE_DILATE = 2;        // cells added around a tile's box
constexpr int TILE_MAX_CELLS = 1024;  // gathered box of cells per tile
constexpr int TILE_MAX_CAND = 1536;   // gathered points per tile (a surface tile gathers ~800)

struct GridStats {
    double sp_sum, sp_cnt;    // spacing pass 1
    double sp2_sum, sp2_cnt;  // spacing pass 2 (trimmed)
    double n_valid;
    double md_sum, md_sq;     // SOR statistics (fixed-order sums)
    float cell, inv_cell;
    int bbox_min[3], bbox_max[3];  // order-preserving float bits
    double thr;                    // SOR threshold, and the largest float <= it
    float thr_f;
    int keep_all;
    unsigned n_deferred;
};

__device__ __forceinline__ int fbits(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float bitsf(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

__device__ __forceinline__ unsigned hash3(int x, int y, int z, unsigned tmask) {
    return ((unsigned)x * 73856093u ^ (unsigned)y * 19349663u ^ (unsigned)z * 83492791u) & tmask;
}

// Deterministic block reduction (fixed shuffle tree); result valid in thread 0.
template <typename T, typename Op>
__device__ __forceinline__ T block_reduce(T v, Op op, T ident) {
    __shared__ T ws[32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int off = 16; off; off >>= 1) v = op(v, __shfl_down_sync(0xffffffffu, v, off));
    if (lane == 0) ws[w] = v;
    __syncthreads();
    T r = ident;
    if (w == 0) {
        r = lane < (int)(blockDim.x >> 5) ? ws[lane] : ident;
        for (int off = 16; off; off >>= 1) r = op(r, __shfl_down_sync(0xffffffffu, r, off));
    }
    __syncthreads();
    return r;
}
struct Add { template <typename T> __device__ T operator()(T a, T b) const { return a + b; } };
struct Min { __device__ int operator()(int a, int b) const { return a < b ? a : b; } };
struct Max { __device__ int operator()(int a, int b) const { return a > b ? a : b; } };

__global__ void stats_init_kernel(GridStats* s) {
    s->sp_sum = s->sp_cnt = s->sp2_sum = s->sp2_cnt = 0;
    for (int a = 0; a < 3; a++) { s->bbox_min[a] = INT_MAX; s->bbox_max[a] = INT_MIN; }
}

// Blocks of the spacing passes (grid-stride).  Each block writes its partial
// sums; spacing_total_kernel adds them in a fixed order, so the cell size does
// not depend on the order blocks finish in.
constexpr int SPACING_BLOCKS = 1024;

// pass 1: mean spacing of horizontally adjacent valid pixels and the bounding
// box.  Counts are integers (exact); a thread's spacings add in FP32 (they only
// set the cell size) and go to FP64 once, for the fixed-order totals.
__global__ void spacing1_kernel(const float* __restrict__ xyz, const uint8_t* __restrict__ mask, int rows, int cols,
                                GridStats* s, double* __restrict__ part) {
    float df = 0.f;
    unsigned ci = 0u;
    int mn[3] = {INT_MAX, INT_MAX, INT_MAX}, mx[3] = {INT_MIN, INT_MIN, INT_MIN};
    // blocks over rows, threads over a row's pixels (no index division), four
    // pixels of a thread at a time with their loads issued together (the same
    // pixels in the same order as one at a time)
    constexpr int U = 4;
    for (int y = blockIdx.x; y < rows; y += gridDim.x) {
        const size_t r0 = (size_t)y * cols;
        for (int xb = threadIdx.x; xb < cols; xb += U * blockDim.x) {
            bool m[U], mr[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int x = xb + u * (int)blockDim.x;
                m[u] = x < cols && mask[r0 + x];
                mr[u] = x + 1 < cols && mask[r0 + x + 1];
            }
            float p[U][3], q[U][3];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const size_t i = r0 + xb + u * blockDim.x;
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    p[u][a] = m[u] ? xyz[3 * i + a] : 0.f;
                    q[u][a] = m[u] && mr[u] ? xyz[3 * i + 3 + a] : 0.f;
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (!m[u] || !zl::finite_point(p[u][0], p[u][1], p[u][2])) continue;
                for (int a = 0; a < 3; a++) {
                    mn[a] = min(mn[a], fbits(p[u][a]));
                    mx[a] = max(mx[a], fbits(p[u][a]));
                }
                if (mr[u] && zl::finite_point(q[u][0], q[u][1], q[u][2])) {
                    float dx = q[u][0] - p[u][0], dy = q[u][1] - p[u][1], dz = q[u][2] - p[u][2];
                    df += sqrtf(dx * dx + dy * dy + dz * dz);
                    ci++;
                }
            }
        }
    }
    double d = block_reduce((double)df, Add(), 0.0);
    double c = block_reduce((double)ci, Add(), 0.0);
    for (int a = 0; a < 3; a++) {
        mn[a] = block_reduce(mn[a], Min(), INT_MAX);
        mx[a] = block_reduce(mx[a], Max(), INT_MIN);
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = d;
        part[2 * blockIdx.x + 1] = c;
        for (int a = 0; a < 3; a++) {
            if (mn[a] != INT_MAX) atomicMin(&s->bbox_min[a], mn[a]);
            if (mx[a] != INT_MIN) atomicMax(&s->bbox_max[a], mx[a]);
        }
    }
}

// pass 2: mean spacing over pairs closer than 3x the pass-1 mean
__global__ void spacing2_kernel(const float* __restrict__ xyz, const uint8_t* __restrict__ mask, int rows, int cols,
                                const GridStats* __restrict__ s, double* __restrict__ part) {
    const double m1 = s->sp_cnt > 0 ? s->sp_sum / s->sp_cnt : 0.0;
    const float cut = (float)(3.0 * m1);  // the pass only sets the cell size
    float df = 0.f;
    unsigned ci = 0u;
    for (int y = blockIdx.x; y < rows; y += gridDim.x)
        for (int x = threadIdx.x; x + 1 < cols; x += blockDim.x) {
            const size_t i = (size_t)y * cols + x;
            if (!(mask[i] && mask[i + 1])) continue;
            float dx = xyz[3 * i + 3] - xyz[3 * i], dy = xyz[3 * i + 4] - xyz[3 * i + 1],
                  dz = xyz[3 * i + 5] - xyz[3 * i + 2];
            float v = sqrtf(dx * dx + dy * dy + dz * dz);
            if (v <= cut) { df += v; ci++; }
        }
    double d = block_reduce((double)df, Add(), 0.0);
    double c = block_reduce((double)ci, Add(), 0.0);
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = d;
        part[2 * blockIdx.x + 1] = c;
    }
}

// Fixed-order total of a spacing pass's block partials (one block of
// SPACING_BLOCKS threads): the mean spacing, then the trimmed mean spacing.
__global__ void spacing_total_kernel(const double* __restrict__ part, int nblk, int pass, GridStats* s) {
    const int t = threadIdx.x;
    double d = t < nblk ? part[2 * t] : 0.0, c = t < nblk ? part[2 * t + 1] : 0.0;
    d = block_reduce(d, Add(), 0.0);
    c = block_reduce(c, Add(), 0.0);
    if (t == 0) {
        (pass == 1 ? s->sp_sum : s->sp2_sum) = d;
        (pass == 1 ? s->sp_cnt : s->sp2_cnt) = c;
    }
}

// Cell = factor * trimmed mean spacing, at least 1e-5 of the cloud's extent (so
// that cell indices stay small).  The size only affects speed, never a result.
__global__ void cell_kernel(GridStats* s, float factor) {
    const double sp = s->sp2_cnt > 0 ? s->sp2_sum / s->sp2_cnt : (s->sp_cnt > 0 ? s->sp_sum / s->sp_cnt : 1.0);
    float cell = (float)(factor * sp), ext = 0.f;
    for (int a = 0; a < 3; a++)
        if (s->bbox_max[a] >= s->bbox_min[a]) ext = fmaxf(ext, bitsf(s->bbox_max[a]) - bitsf(s->bbox_min[a]));
    cell = fmaxf(cell, ext * 1e-5f);
    cell = fmaxf(cell, 1e-6f);
    s->cell = cell;
    s->inv_cell = 1.0f / cell;
}

// Squared distance with one fixed rounding sequence, so the same pair of
// points gives the same value at every call site of the kNN search.
__device__ __forceinline__ float sqdist(float dx, float dy, float dz) { return fmaf(dz, dz, fmaf(dy, dy, dx * dx)); }

// Hardware square root (PTX sqrt.approx.f32, relative error below 2^-22): one
// instruction, the same at every call site, so every search path rounds alike.
__device__ __forceinline__ float root_approx(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Order-independent sum of the k + 1 nearest distances: each root, scaled by
// 2^(23 - e) with root(largest squared distance) < 2^e, is truncated to an
// integer below 2^23 and the integers are added exactly (at most 64 of them:
// below 2^29), so every search path and every visiting order gives the same
// bits.  The truncation is one FMA rounded toward zero onto 2^23, whose
// mantissa then holds the integer: no 64-bit conversion (FP64 pipe) per root.
// The roots are root_approx's; e leaves 2^-19 of room above the largest, more
// than the approximation's error, so no smaller entry's root reaches 2^e.
// Roots below 2^(e - 23), a 2^-22 fraction of the largest, count as 0.
__device__ __forceinline__ int root_exponent(float d2max) {
    int e;
    frexpf(root_approx(d2max) * 1.000002f, &e);
    return min(max(e, -60), 100);  // keeps 2^(23 - e) and 2^(e - 23) normal
}
__device__ __forceinline__ float root_scale(int e) { return __uint_as_float((unsigned)(150 - e) << 23); }
__device__ __forceinline__ unsigned root_fixed(float d2, float scale) {
    return __float_as_uint(__fmaf_rz(root_approx(d2), scale, 8388608.f)) - 0x4B000000u;
}
// (sum / k) 2^(e - 23), one float division
__device__ __forceinline__ float fixed_mean(unsigned sum, int e, int k) {
    return __fdiv_rn(__uint2float_rn(sum), (float)k) * __uint_as_float((unsigned)(104 + e) << 23);
}

__device__ __forceinline__ void cell_of(float x, float y, float z, float ic, int& cx, int& cy, int& cz) {
    cx = __float2int_rd(x * ic);
    cy = __float2int_rd(y * ic);
    cz = __float2int_rd(z * ic);
}

__device__ __forceinline__ unsigned grid_slot(const GridStats* __restrict__ s, unsigned tmask, float x, float y,
                                              float z) {
    int cx, cy, cz;
    cell_of(x, y, z, s->inv_cell, cx, cy, cz);
    return hash3(cx, cy, cz, tmask);
}

// Neighbouring pixels mostly share a cell, so the lanes of a warp that hit the
// same slot add to it once (the lowest such lane).
// The table kernels stride over the points with a grid sized to the GPU.
__global__ void hash_count_kernel(const float* __restrict__ xyz, const uint8_t* __restrict__ mask, size_t n,
                                  const GridStats* __restrict__ s, unsigned tmask,
                                  unsigned* __restrict__ counts) {
    for (size_t b = (size_t)blockIdx.x * blockDim.x; b < n; b += (size_t)gridDim.x * blockDim.x) {
        const size_t i = b + threadIdx.x;
        const bool v = i < n && mask[i] && zl::finite_point(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]);
        const unsigned h = v ? grid_slot(s, tmask, xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]) : 0xffffffffu;
        const unsigned grp = __match_any_sync(0xffffffffu, h);
        if (v && (threadIdx.x & 31) == __ffs(grp) - 1) atomicAdd(&counts[h], (unsigned)__popc(grp));
    }
}

__global__ void zero_kernel(unsigned* __restrict__ p, size_t n) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        p[i] = 0u;
}

__device__ __forceinline__ unsigned block_scan_incl(unsigned v, unsigned* ws) {
    unsigned x = v;
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int off = 1; off < 32; off <<= 1) {
        unsigned t = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += t;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
        unsigned y = ws[lane];
        for (int off = 1; off < 32; off <<= 1) {
            unsigned t = __shfl_up_sync(0xffffffffu, y, off);
            if (lane >= off) y += t;
        }
        ws[lane] = y;
    }
    __syncthreads();
    return x + (w ? ws[w - 1] : 0u);
}

// exclusive scan of the counts into tab[].x (per-block part), block totals
__global__ void scan_blocks_kernel(const unsigned* __restrict__ counts, uint2* __restrict__ tab, size_t n,
                                   unsigned* __restrict__ block_tot) {
    __shared__ unsigned ws[32];
    const size_t nb = (n + SCAN_B - 1) / SCAN_B;
    for (size_t b = blockIdx.x; b < nb; b += gridDim.x) {
        const size_t i = b * SCAN_B + threadIdx.x;
        const unsigned v = i < n ? counts[i] : 0u;
        const unsigned incl = block_scan_incl(v, ws);
        if (i < n) tab[i] = make_uint2(incl - v, v);
        if (threadIdx.x == SCAN_B - 1) block_tot[b] = incl;
        __syncthreads();  // ws is reused by the next chunk
    }
}

__global__ void scan_totals_kernel(unsigned* __restrict__ tot, int nb) {
    __shared__ unsigned carry;
    __shared__ unsigned ws[32];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nb; base += SCAN_B) {
        int i = base + threadIdx.x;
        unsigned v = i < nb ? tot[i] : 0u;
        unsigned incl = block_scan_incl(v, ws);
        unsigned c = carry;
        if (i < nb) tot[i] = c + incl - v;
        __syncthreads();
        if (threadIdx.x == SCAN_B - 1) carry = c + incl;
        __syncthreads();
    }
}

__global__ void scan_add_kernel(uint2* __restrict__ tab, size_t n, const unsigned* __restrict__ tot) {
    const size_t nb = (n + SCAN_B - 1) / SCAN_B;
    for (size_t b = blockIdx.x; b < nb; b += gridDim.x) {
        const size_t i = b * SCAN_B + threadIdx.x;
        if (i < n) tab[i].x += tot[b];
    }
}

__global__ void hash_scatter_kernel(const float* __restrict__ xyz, const uint8_t* __restrict__ mask, size_t n,
                                    const GridStats* __restrict__ s, unsigned tmask,
                                    const uint2* __restrict__ tab, unsigned* __restrict__ fill,
                                    float4* __restrict__ pts) {
    for (size_t b = (size_t)blockIdx.x * blockDim.x; b < n; b += (size_t)gridDim.x * blockDim.x) {
        const size_t i = b + threadIdx.x;
        const bool v = i < n && mask[i] && zl::finite_point(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]);
        float x = 0.f, y = 0.f, z = 0.f;
        unsigned h = 0xffffffffu;
        if (v) {
            x = xyz[3 * i]; y = xyz[3 * i + 1]; z = xyz[3 * i + 2];
            h = grid_slot(s, tmask, x, y, z);
        }
        // one atomic per slot and warp; lanes take consecutive places in lane order
        const unsigned grp = __match_any_sync(0xffffffffu, h);
        const int lane = threadIdx.x & 31, leader = __ffs(grp) - 1;
        unsigned base = 0;
        if (v && lane == leader) base = atomicAdd(&fill[h], (unsigned)__popc(grp));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (v) {
            const unsigned pos = tab[h].x + base + (unsigned)__popc(grp & ((1u << lane) - 1u));
            pts[pos] = make_float4(x, y, z, __int_as_float((int)i));
        }
    }
}

struct Level {
    const uint2* tab;  // (offset, count) per bucket
    const float4* pts;
    unsigned tmask;
};

__device__ __forceinline__ uint2 bucket(const Level& g, int x, int y, int z) {
    return __ldg(g.tab + hash3(x, y, z, g.tmask));
}

// Pixel offsets within WIN_R of the centre, ordered by length.
constexpr int WIN_R = 4;
constexpr int WIN_W = TILE_X + 2 * WIN_R, WIN_H = TILE_Y + 2 * WIN_R;
constexpr int WIN_N = (2 * WIN_R + 1) * (2 * WIN_R + 1) - 1;
__constant__ signed char c_spiral[WIN_N][2] = {
    {0, -1}, {-1, 0}, {1, 0}, {0, 1}, {-1, -1}, {1, -1}, {-1, 1}, {1, 1}, {0, -2}, {-2, 0},
    {2, 0}, {0, 2}, {-1, -2}, {1, -2}, {-2, -1}, {2, -1}, {-2, 1}, {2, 1}, {-1, 2}, {1, 2},
    {-2, -2}, {2, -2}, {-2, 2}, {2, 2}, {0, -3}, {-3, 0}, {3, 0}, {0, 3}, {-1, -3}, {1, -3},
    {-3, -1}, {3, -1}, {-3, 1}, {3, 1}, {-1, 3}, {1, 3}, {-2, -3}, {2, -3}, {-3, -2}, {3, -2},
    {-3, 2}, {3, 2}, {-2, 3}, {2, 3}, {0, -4}, {-4, 0}, {4, 0}, {0, 4}, {-1, -4}, {1, -4},
    {-4, -1}, {4, -1}, {-4, 1}, {4, 1}, {-1, 4}, {1, 4}, {-3, -3}, {3, -3}, {-3, 3}, {3, 3},
    {-2, -4}, {2, -4}, {-4, -2}, {4, -2}, {-4, 2}, {4, 2}, {-2, 4}, {2, 4}, {-3, -4}, {3, -4},
    {-4, -3}, {4, -3}, {-4, 3}, {4, 3}, {-3, 4}, {3, 4}, {-4, -4}, {4, -4}, {-4, 4}, {4, 4}};
static_assert(WIN_W * WIN_H <= TILE_MAX_CAND, "pixel window staged in the candidate buffer");
static_assert(TILE_MAX_CELLS <= 8 * TILE_T, "cell scan: eight cells per thread");

constexpr int SV_CAP = 128;  // survivors per warp query (k + 1 <= 64 of them kept)

// Tile search: one CTA per 16 x 8 pixel tile on the grid.
//  - Window bound: the query and its k nearest valid pixels (in pixel
//    distance, within WIN_R) are k + 1 real points, so the largest of their
//    squared distances, tau0, bounds the (k + 1)-th nearest squared distance.
//  - Box: the tile's points, minus depth outliers (a trimmed mean of their z
//    cells), span a box of cells; the CTA gathers every point of that box
//    dilated by TILE_DILATE cells into shared memory, sorted by cell.  All
//    points within distance g of a query lie in the box, g being the query's
//    distance to the box boundary.
//  - Each in-box query scans only the cells its ball of squared radius
//    min(tau0, g^2) touches; holding k + 1 candidates within that ball, it is
//    exact.  The warp does this one query at a time, lanes over candidates.
// Queries the box cannot settle search the cells that hold the
// ball of radius sqrt(tau0) (up to FINE_RINGS rings).  Unresolved queries are
// appended to the deferred list with md = -1.  (Clouds with pixel rays skip
// this phase: the window passes take every query.)
__global__ void __launch_bounds__(TILE_T) sor_knn_tile_kernel(const float* __restrict__ xyz,
                                                              const uint8_t* __restrict__ mask, int rows, int cols,
                                                              int k, Level g, const GridStats* __restrict__ s, zl::Head* h,
                                                              float* __restrict__ md_out,
                                                              unsigned* __restrict__ deferred) {
    extern __shared__ float4 tile_smem[];
    float4* cand = tile_smem;                  // TILE_MAX_CAND
    __shared__ int s_off[TILE_MAX_CELLS + 1];  // candidate offset of each box cell
    __shared__ float s_sv[TILE_T / 32 * SV_CAP];  // per-warp survivor lists
    __shared__ int s_nsv[TILE_T / 32];
    __shared__ unsigned s_ws[32];
    __shared__ int s_box[6];
    __shared__ float s_zc;
    __shared__ unsigned s_total;
    const int tid = threadIdx.x;
    const int x0 = blockIdx.x * TILE_X, y0 = blockIdx.y * TILE_Y;
    const int x = x0 + (tid % TILE_X), y = y0 + (tid / TILE_X);
    const bool in = x < cols && y < rows;
    const size_t i = in ? (size_t)y * cols + x : 0;
    const bool valid = in && mask[i] && h->n_valid > (unsigned)k;
    if (in && !valid) md_out[i] = 0.f;
    if (!__syncthreads_or(valid)) return;  // the whole CTA leaves together
    const float ic = s->inv_cell, cell = s->cell;
    float qx = 0.f, qy = 0.f, qz = 0.f;
    int c[3] = {0, 0, 0};
    bool active = false;  // a query without finite coordinates is not searched here
    if (valid) {
        qx = xyz[3 * i]; qy = xyz[3 * i + 1]; qz = xyz[3 * i + 2];
        active = zl::finite_point(qx, qy, qz);
    }
    if (active) cell_of(qx, qy, qz, ic, c[0], c[1], c[2]);
    // window bound tau0 from the pixel neighbourhood (staged in cand; w = 0 marks
    // pixels without a finite point)
    for (int t = tid; t < WIN_W * WIN_H; t += TILE_T) {
        const int wx = x0 - WIN_R + t % WIN_W, wy = y0 - WIN_R + t / WIN_W;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (wx >= 0 && wx < cols && wy >= 0 && wy < rows) {
            const size_t j = (size_t)wy * cols + wx;
            const float px = xyz[3 * j], py = xyz[3 * j + 1], pz = xyz[3 * j + 2];
            if (mask[j] && zl::finite_point(px, py, pz)) v = make_float4(px, py, pz, 1.f);
        }
        cand[t] = v;
    }
    __syncthreads();
    float tau0 = INFINITY;
    if (active) {
        const int wc = (tid / TILE_X + WIN_R) * WIN_W + tid % TILE_X + WIN_R;
        int found = 0;
        float m = 0.f;
        for (int o = 0; o < WIN_N && found < k; o++) {
            const float4 p = cand[wc + c_spiral[o][1] * WIN_W + c_spiral[o][0]];
            if (p.w == 0.f) continue;
            const float dx = p.x - qx, dy = p.y - qy, dz = p.z - qz;
            m = fmaxf(m, sqdist(dx, dy, dz));
            found++;
        }
        if (found == k) tau0 = m;
    }
    __syncthreads();
    // trimmed mean of the z cells: mean, then mean of those within 8 cells of it
    float n1 = block_reduce(active ? 1.f : 0.f, Add(), 0.f);
    float z1 = block_reduce(active ? (float)c[2] : 0.f, Add(), 0.f);
    if (tid == 0) s_zc = n1 > 0 ? z1 / n1 : 0.f;
    __syncthreads();
    bool near1 = active && fabsf((float)c[2] - s_zc) <= 8.f;
    float n2 = block_reduce(near1 ? 1.f : 0.f, Add(), 0.f);
    float z2 = block_reduce(near1 ? (float)c[2] : 0.f, Add(), 0.f);
    __syncthreads();
    if (tid == 0) s_zc = n2 > 0 ? z2 / n2 : s_zc;
    __syncthreads();
    const bool inbox = active && fabsf((float)c[2] - s_zc) <= 4.f;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        int lo = block_reduce(inbox ? c[a] : INT_MAX, Min(), INT_MAX);
        int hi = block_reduce(inbox ? c[a] : INT_MIN, Max(), INT_MIN);
        if (tid == 0) { s_box[a] = lo; s_box[3 + a] = hi; }
    }
    __syncthreads();
    const bool any = s_box[0] != INT_MAX;
    const int lo0 = s_box[0] - TILE_DILATE, lo1 = s_box[1] - TILE_DILATE, lo2 = s_box[2] - TILE_DILATE;
    const long long ex = any ? (long long)s_box[3] - s_box[0] + 1 + 2 * TILE_DILATE : 0;
    const long long ey = any ? (long long)s_box[4] - s_box[1] + 1 + 2 * TILE_DILATE : 0;
    const long long ez = any ? (long long)s_box[5] - s_box[2] + 1 + 2 * TILE_DILATE : 0;
    const long long V = ex * ey * ez;
    bool fast = any && V <= TILE_MAX_CELLS;  // uniform over the CTA
    if (fast) {
        // counting sort of the box's points by cell: count, scan, place
        for (int t = tid; t < V; t += TILE_T) {
            const int ix = lo0 + (int)(t % ex), iy = lo1 + (int)((t / ex) % ey), iz = lo2 + (int)(t / (ex * ey));
            const uint2 b = bucket(g, ix, iy, iz);
            int n_in = 0;
            for (unsigned u = b.x; u < b.x + b.y; u++) {
                const float4 p = __ldg(g.pts + u);
                int px, py, pz;
                cell_of(p.x, p.y, p.z, ic, px, py, pz);
                n_in += (px == ix && py == iy && pz == iz);
            }
            s_off[t] = n_in;
        }
        __syncthreads();
        unsigned v8[8], own = 0;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int t = tid * 8 + u;
            v8[u] = t < V ? (unsigned)s_off[t] : 0u;
            own += v8[u];
        }
        const unsigned incl = block_scan_incl(own, s_ws);
        unsigned run = incl - own;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int t = tid * 8 + u;
            if (t < V) s_off[t] = (int)run;
            run += v8[u];
        }
        if (tid == TILE_T - 1) {
            s_total = incl;
            s_off[V] = (int)incl;
        }
        __syncthreads();
        fast = s_total <= (unsigned)TILE_MAX_CAND;
        if (fast) {
            for (int t = tid; t < V; t += TILE_T) {
                const int ix = lo0 + (int)(t % ex), iy = lo1 + (int)((t / ex) % ey), iz = lo2 + (int)(t / (ex * ey));
                const uint2 b = bucket(g, ix, iy, iz);
                int pos = s_off[t];
                for (unsigned u = b.x; u < b.x + b.y; u++) {
                    const float4 p = __ldg(g.pts + u);
                    int px, py, pz;
                    cell_of(p.x, p.y, p.z, ic, px, py, pz);
                    if (px == ix && py == iy && pz == iz) cand[pos++] = p;
                }
            }
        }
        __syncthreads();
    }
    const int K1 = k + 1;
    const bool fq = active && fast && inbox;
    // margin for the float rounding of the cell mapping (|p| * 2^-23 << 1e-3 cell)
    const float margin = fmaxf(1e-3f * cell, 4e-7f * fmaxf(fabsf(qx), fmaxf(fabsf(qy), fabsf(qz))));
    float thr = -1.f;
    int bx0 = INT_MAX, by0 = INT_MAX, bz0 = INT_MAX, bx1 = INT_MIN, by1 = INT_MIN, bz1 = INT_MIN;
    if (fq) {
        float gmin = fminf(fminf(qx - lo0 * cell, (lo0 + ex) * cell - qx),
                           fminf(fminf(qy - lo1 * cell, (lo1 + ey) * cell - qy),
                                 fminf(qz - lo2 * cell, (lo2 + ez) * cell - qz)));
        gmin = fmaxf(gmin - margin, 0.f);
        // every point with d2 <= thr lies in the cells the ball of radius R touches
        thr = fminf(tau0, gmin * gmin);
        const float R = sqrtf(thr) + margin;
        bx0 = max(lo0, __float2int_rd((qx - R) * ic)); bx1 = min(lo0 + (int)ex - 1, __float2int_rd((qx + R) * ic));
        by0 = max(lo1, __float2int_rd((qy - R) * ic)); by1 = min(lo1 + (int)ey - 1, __float2int_rd((qy + R) * ic));
        bz0 = max(lo2, __float2int_rd((qz - R) * ic)); bz1 = min(lo2 + (int)ez - 1, __float2int_rd((qz + R) * ic));
    }
    // Warp-cooperative selection, one query at a time: the lanes split the
    // query's candidate cells, keep the squared distances within its bound in
    // the warp's survivor list, then drop the largest until k + 1 remain and
    // sum their roots in fixed point (the same bits on every path).
    //  - fast queries read the cell-sorted box in shared memory (consecutive
    //    lanes, consecutive candidates);
    //  - the others (and fast queries the box could not settle) search the
    //    rings of cells that hold the ball of their window bound tau0,
    //    one cell per lane from the global table;
    //  - what neither settles is deferred to the tree search with md = -1.
    const unsigned full = 0xffffffffu;
    const int lane = tid & 31, wid = tid >> 5;
    float* sv = s_sv + wid * SV_CAP;
    bool done = false;
    // rings that hold every point within sqrt(tau0) of the query (|floor a - floor b| <= ceil |a - b|)
    int rr = INT_MAX;
    if (active && tau0 < INFINITY) rr = (int)ceilf((sqrtf(tau0) + margin) * ic);
    for (int pass = 0; pass < 2; pass++) {
        unsigned todo = __ballot_sync(full, pass == 0 ? fq : (active && !done && rr <= FINE_RINGS));
        while (todo) {
            const int q = __ffs(todo) - 1;
            todo &= todo - 1;
            const float Qx = __shfl_sync(full, qx, q), Qy = __shfl_sync(full, qy, q), Qz = __shfl_sync(full, qz, q);
            const float T = __shfl_sync(full, pass == 0 ? thr : tau0, q);
            int nsv = 0;
            if (pass == 0) {
                const int X0 = __shfl_sync(full, bx0, q), X1 = __shfl_sync(full, bx1, q);
                const int Y0 = __shfl_sync(full, by0, q), Y1 = __shfl_sync(full, by1, q);
                const int Z0 = __shfl_sync(full, bz0, q), Z1 = __shfl_sync(full, bz1, q);
                for (int iz = Z0; iz <= Z1; iz++)
                    for (int iy = Y0; iy <= Y1; iy++) {
                        const int row = (int)(((long long)(iz - lo2) * ey + (iy - lo1)) * ex) - lo0;
                        const int j0 = s_off[row + X0], j1 = s_off[row + X1 + 1];
                        for (int jb = j0; jb < j1; jb += 32) {
                            const int j = jb + lane;
                            float d2 = INFINITY;
                            if (j < j1) {
                                const float4 p = cand[j];
                                d2 = sqdist(p.x - Qx, p.y - Qy, p.z - Qz);
                            }
                            const bool keep = d2 <= T;
                            const unsigned b = __ballot_sync(full, keep);
                            const int pos = nsv + __popc(b & ((1u << lane) - 1u));
                            if (keep && pos < SV_CAP) sv[pos] = d2;
                            nsv += __popc(b);
                        }
                    }
            } else {
                const int C0 = __shfl_sync(full, c[0], q), C1 = __shfl_sync(full, c[1], q);
                const int C2 = __shfl_sync(full, c[2], q), R = __shfl_sync(full, rr, q);
                const int side = 2 * R + 1, ncell = side * side * side;
                if (lane == 0) s_nsv[wid] = 0;
                __syncwarp();
                for (int t = lane; t < ncell; t += 32) {
                    const int cx = C0 - R + t % side, cy = C1 - R + (t / side) % side, cz = C2 - R + t / (side * side);
                    const uint2 b = bucket(g, cx, cy, cz);
                    for (unsigned u = b.x; u < b.x + b.y; u++) {
                        const float4 p = __ldg(g.pts + u);
                        int px, py, pz;
                        cell_of(p.x, p.y, p.z, ic, px, py, pz);
                        if (px != cx || py != cy || pz != cz) continue;
                        const float d2 = sqdist(p.x - Qx, p.y - Qy, p.z - Qz);
                        if (d2 > T) continue;
                        const int pos = atomicAdd(&s_nsv[wid], 1);
                        if (pos < SV_CAP) sv[pos] = d2;
                    }
                }
                __syncwarp();
                nsv = s_nsv[wid];
            }
            __syncwarp();
            if (nsv < K1 || nsv > SV_CAP) continue;  // warp-uniform: not settled here
            // keys: squared-distance bits + 1 (non-negative floats order as unsigned); 0 = empty
            unsigned key[SV_CAP / 32];
#pragma unroll
            for (int r = 0; r < SV_CAP / 32; r++) {
                const int idx = lane + 32 * r;
                key[r] = idx < nsv ? __float_as_uint(sv[idx]) + 1u : 0u;
            }
            for (int m = nsv - K1; m > 0; m--) {
                unsigned lm = 0;
#pragma unroll
                for (int r = 0; r < SV_CAP / 32; r++) lm = max(lm, key[r]);
                const unsigned wm = __reduce_max_sync(full, lm);
                const unsigned own = __ballot_sync(full, lm == wm);
                if (lane == __ffs(own) - 1) {
                    bool gone = false;
#pragma unroll
                    for (int r = 0; r < SV_CAP / 32; r++)
                        if (!gone && key[r] == wm) { key[r] = 0u; gone = true; }
                }
            }
            unsigned lm = 0;
#pragma unroll
            for (int r = 0; r < SV_CAP / 32; r++) lm = max(lm, key[r]);
            const float vmax = __uint_as_float(__reduce_max_sync(full, lm) - 1u);
            const int e = root_exponent(vmax);
            const float sc = root_scale(e);
            unsigned part = 0;
#pragma unroll
            for (int r = 0; r < SV_CAP / 32; r++)
                if (key[r]) part += root_fixed(__uint_as_float(key[r] - 1u), sc);
            part = __reduce_add_sync(full, part);
            if (lane == q) {
                md_out[i] = fixed_mean(part, e, k);
                done = true;
            }
        }
    }
    if (valid && !done) {
        md_out[i] = -1.f;
        const unsigned slot = atomicAdd(&h->n_deferred, 1u);
        deferred[slot] = (unsigned)i;
    }
}

// ------------------------------------------------ window fast path (SOR) ----
//
// An organised cloud from one camera keeps its neighbours close in the image:
// a point p seen along the ray of pixel b, and a query q near the ray of pixel
// a, satisfy |p - q| >= |q| sin(angle(a, b)) - dev(q) - dev(p), where dev is a
// point's distance from its own pixel ray.  For every pixel b outside the
// (2 WR + 1)^2 window around a, |b - a| >= WR + 1 pixels, and with the pinhole
// rays a = (u - cx, v - cy, f), |a x b| >= f |b - a| and |b| <= |a| + |b - a|,
// so sin(angle) >= f (WR + 1) / (|a| (|a| + WR + 1)).  A query whose k + 1
// nearest points inside its window lie within
//     |q| f (WR + 1) / (|a| (|a| + WR + 1)) - dev(q) - max dev
// has the same k + 1 nearest points in the whole cloud: its mean distance is
// exact from the window alone.  Inside the window the same bound holds with the
// largest dev of the block's staged points in place of the cloud's (points
// averaged across a depth edge lie far off their rays, but only near it), so
// the spiral stops at the radius that local bound gives and the cloud-wide
// maximum only has to clear the window's edge.  Queries the bounds do not
// certify go to the deferred list (md = -1) for the tree search.

using zt::RayParams;
using zt::ray_dir;
using zt::ray_dev;
constexpr int WR = zt::SPIRAL_R;  // window half-size of the fast path
constexpr int WW = WT_X + 2 * WR, WH = WT_Y + 2 * WR;
constexpr int WN = zt::SPIRAL_N;
constexpr int WR2MAX = 2 * WR * WR;

// The window's pixel offsets ordered by length, then row, then column, as
// staged-tile offsets with their squared length, and per squared radius the
// number of offsets within it: a walk's stop radius becomes a loop limit.
struct WinSpiral {
    int ent[WN];             // (dy * WW + dx) & 0xffff | (dx^2 + dy^2) << 16
    short upto[WR2MAX + 1];  // offsets of squared length <= i
    constexpr WinSpiral() : ent(), upto() {
        int n = 0;
        for (int l = 1; l <= WR2MAX; l++)
            for (int dy = -WR; dy <= WR; dy++)
                for (int dx = -WR; dx <= WR; dx++)
                    if (dx * dx + dy * dy == l) ent[n++] = ((dy * WW + dx) & 0xffff) | (l << 16);
        int c = 0;
        for (int i = 0; i <= WR2MAX; i++) {
            while (c < WN && (ent[c] >> 16) <= i) c++;
            upto[i] = (short)c;
        }
    }
};
__constant__ WinSpiral c_win = WinSpiral();
constexpr WinSpiral k_win{};  // the same table at compile time
// tile offset of spiral entry O as a compile-time constant
template <int O>
__device__ __forceinline__ int win_off_c() {
    constexpr int v = (int)(short)(k_win.ent[O] & 0xffff);
    return v;
}
__device__ __forceinline__ int win_off(int o) { return (int)(short)(c_win.ent[o] & 0xffff); }
__device__ __forceinline__ int win_len2(int o) { return c_win.ent[o] >> 16; }
// offsets whose squared length is at most r2 (r2 >= 0 or +inf)
__device__ __forceinline__ int win_upto(float r2) { return r2 < (float)WR2MAX ? c_win.upto[(int)r2] : WN; }

// The k + 1 smallest squared distances a thread has seen, in G groups of five: a
// group's largest in a register, the other four as one float4 in column tid of a
// [G][WT_T] shared array (conflict-free).  The largest of all is the largest of
// the registers; a nearer point takes its place, and one pass over its group finds
// the group's next largest.  Unused places hold 0, the query's own distance: never
// the largest unless all are 0, and no part of a sum of roots.
//
// A binary heap in shared memory took its place, five or six dependent loads deep
// per replacement and with a build besides.  Window pass, k = 50, 1280 x 1024: 234
// -> 150 us; k = 20: 127 -> 79 us.  Groups of nine take two loads and fewer
// registers, but hold fewer CTAs at k = 50 (688 against 660 us for the whole filter
// of a 2448 x 2048 cloud); at the other k they are even.
constexpr int NS_N = 5;  // values per group
template <int G>
struct NearSet {
    float4* S;
    float top[G];
    // the larger of t and e stays in t
    static __device__ __forceinline__ void order(float& e, float& t) {
        const float lo = fminf(e, t);
        t = fmaxf(e, t);
        e = lo;
    }
    __device__ __forceinline__ float largest() const {
        float m = top[0];
#pragma unroll
        for (int g = 1; g < G; g++) m = fmaxf(m, top[g]);
        return m;
    }
    // v in the place of the largest (m = largest())
    __device__ __forceinline__ void replace(float v, float m) {
        int g = 0;
#pragma unroll
        for (int j = 1; j < G; j++) g = top[j] == m ? j : g;
        float4 a = S[g * WT_T];
        order(a.x, v);
        order(a.y, v);
        order(a.z, v);
        order(a.w, v);
        S[g * WT_T] = a;
#pragma unroll
        for (int j = 0; j < G; j++) top[j] = j == g ? v : top[j];
    }
};

// A query the window pass cannot settle goes straight to the deferred list
// (md = -1) for the tree search.
__device__ __forceinline__ void defer_query(zl::Head* h, unsigned* deferred, float* md_out, size_t i) {
    md_out[i] = -1.f;
    deferred[atomicAdd(&h->n_deferred, 1u)] = (unsigned)i;
}

// The same with an upper bound on its (k + 1)-th smallest squared distance
// (md = MD_BOUND, the bound in `bound`): the tree search starts from it.
__device__ __forceinline__ void defer_query_bound(zl::Head* h, unsigned* deferred, float* md_out, float* bound,
                                                  size_t i, float b) {
    bound[i] = b;
    md_out[i] = MD_BOUND;
    deferred[atomicAdd(&h->n_deferred, 1u)] = (unsigned)i;
}

// The window pass's staged points: coordinates in two arrays (12 bytes a point
// hold one CTA more per SM than 16), +inf for an invalid pixel's.
constexpr size_t WIN_BYTES = (size_t)WW * WH * 12;
static_assert(WIN_BYTES % 16 == 0, "the sets behind the window are float4");
struct WinPoints {
    float2* xy;
    float* z;
    __device__ __forceinline__ float d2(int e, float x, float y, float zq) const {
        const float2 p = xy[e];
        return sqdist(p.x - x, p.y - y, z[e] - zq);
    }
};

// Group g of the set: spiral offsets 5 g to 5 g + 4, in the last group those below k.
template <int G, int g, int... J>
__device__ __forceinline__ void fill_group(NearSet<G>& set, const WinPoints& W, int wc, float qx, float qy, float qz,
                                           int k, std::integer_sequence<int, J...>) {
    float v[NS_N] = {(g + 1 < G || NS_N * g + J < k ? W.d2(wc + win_off_c<NS_N * g + J>(), qx, qy, qz) : 0.f)...};
    float t = v[NS_N - 1];
#pragma unroll
    for (int j = 0; j < NS_N - 1; j++) NearSet<G>::order(v[j], t);
    set.S[g * WT_T] = make_float4(v[0], v[1], v[2], v[3]);
    set.top[g] = t;
}
template <int G, int... g>
__device__ __forceinline__ void fill_groups(NearSet<G>& set, const WinPoints& W, int wc, float qx, float qy, float qz,
                                            int k, std::integer_sequence<int, g...>) {
    (fill_group<G, g>(set, W, wc, qx, qy, qz, k, std::make_integer_sequence<int, NS_N>{}), ...);
}

// G: groups of the set, (k + 1) / NS_N rounded up
template <int G>
__global__ void __launch_bounds__(WT_T) sor_window_kernel(const float* __restrict__ xyz,
                                                            const uint8_t* __restrict__ mask, int rows, int cols,
                                                            int k, RayParams rp, zl::Tree t,
                                                            float* __restrict__ md_out,
                                                            unsigned* __restrict__ deferred,
                                                            float* __restrict__ bound) {
    extern __shared__ float4 win_smem[];
    const WinPoints W{reinterpret_cast<float2*>(win_smem),
                      reinterpret_cast<float*>(reinterpret_cast<float2*>(win_smem) + WW * WH)};
    const int tid = threadIdx.x;
    const int x0 = blockIdx.x * WT_X, y0 = blockIdx.y * WT_Y;
    zl::Head* h = t.head;
    // largest ray distance of the leaves that the window touches (float bits, >= 0)
    __shared__ unsigned win_dev;
    if (tid < 32) {
        const int lx0 = max(x0 - WR, 0) / zl::LEAF, lx1 = min((x0 + WT_X - 1 + WR) / zl::LEAF, t.lw - 1);
        const int ly0 = max(y0 - WR, 0) / zl::LEAF, ly1 = min((y0 + WT_Y - 1 + WR) / zl::LEAF, t.lh - 1);
        const int nx = lx1 - lx0 + 1;
        unsigned d = 0u;
        for (int e = tid; e < nx * (ly1 - ly0 + 1); e += 32)
            d = max(d, __float_as_uint(__ldg(t.leaf + 2 * ((size_t)(ly0 + e / nx) * t.lw + lx0 + e % nx) + 1).w));
        d = __reduce_max_sync(0xffffffffu, d);
        if (tid == 0) win_dev = d;
    }
#pragma unroll
    for (int e = tid; e < WW * WH; e += WT_T) {
        const int wx = x0 - WR + e % WW, wy = y0 - WR + e / WW;
        // invalid and off-image pixels and points without finite coordinates at
        // +inf: nearer than no point
        float2 vxy = make_float2(INFINITY, INFINITY);
        float vz = INFINITY;
        if (wx >= 0 && wx < cols && wy >= 0 && wy < rows) {
            const size_t j = (size_t)wy * cols + wx;
            const float px = xyz[3 * j], py = xyz[3 * j + 1], pz = xyz[3 * j + 2];
            if (mask[j] && fabsf(px) + fabsf(py) + fabsf(pz) < INFINITY) {
                vxy = make_float2(px, py);
                vz = pz;
            }
        }
        W.xy[e] = vxy;
        W.z[e] = vz;
    }
    __syncthreads();
    const unsigned tdev = win_dev;
    const int tx = tid % WT_X, ty = tid / WT_X;
    const int x = x0 + tx, y = y0 + ty;
    if (x >= cols || y >= rows) return;  // no block-wide synchronisation below
    const size_t i = (size_t)y * cols + x;
    if (!mask[i] || !(h->n_valid > (unsigned)k)) {
        md_out[i] = 0.f;
        return;
    }
    const int wc = (ty + WR) * WW + tx + WR;
    const float qx = W.xy[wc].x, qy = W.xy[wc].y, qz = W.z[wc];
    if (!(qx < INFINITY)) {
        defer_query(h, deferred, md_out, i);
        return;
    }
    // the query and its first k window pixels in spiral order fill the set, an
    // invalid pixel at +inf (the first valid distance to come replaces it; a set
    // still holding one at the end means fewer than k + 1 points)
    NearSet<G> set;
    set.S = win_smem + WIN_BYTES / 16 + tid;
    fill_groups<G>(set, W, wc, qx, qy, qz, k, std::make_integer_sequence<int, G>{});
    int o = k;
    float thr = set.largest();
    // bound(r) = C r / (an + r): no point of a pixel at distance >= r from the
    // query's lies nearer than bound(r) - dev (slack: float rounding, 1e-5 |q|)
    float ax, ay, az;
    ray_dir(rp, x, y, ax, ay, az);
    const float an = sqrtf(fmaf(ax, ax, fmaf(ay, ay, az * az)));
    const float qn = sqrtf(fmaf(qx, qx, fmaf(qy, qy, qz * qz)));
    const float C = qn * rp.f / an;
    const float dev_q = ray_dev(qx, qy, qz, ax, ay, az) + 1e-5f * qn;
    const float dev = dev_q + __uint_as_float(tdev);                    // window pixels
    const float dev_out = dev_q + __uint_as_float(h->ray_dev_bits);     // pixels outside it
    // squared pixel distance beyond which every window point is farther than
    // sqrt(thr): C r / (an + r) > sqrt(thr) + dev  <=>  r > (sqrt(thr) + dev) an / (C - sqrt(thr) - dev).
    // Approximate arithmetic: the stop only ends the walk; the exact
    // certificate below decides whether the window result stands.
    auto stop_r2 = [&](float thr) {
        const float sd = root_approx(thr) + dev;
        if (!(C > sd)) return INFINITY;
        const float r = __fdividef(sd * an, C - sd);
        return r * r;
    };
    // the spiral runs by increasing length: once past the stop distance, the
    // rest of the window (and everything outside it) is provably farther
    int lim = win_upto(stop_r2(thr));
    auto at = [&](int o) { return o < WN ? W.d2(wc + win_off(o), qx, qy, qz) : INFINITY; };
    for (; o < lim; o += 4) {
        float d0 = at(o), d1 = at(o + 1), d2 = at(o + 2), d3 = at(o + 3);
        if (!(fminf(fminf(d0, d1), fminf(d2, d3)) < thr)) continue;
        // one replacement of every lane that has any, until none has
        for (;;) {
            const bool c0 = d0 < thr, c1 = d1 < thr, c2 = d2 < thr, c3 = d3 < thr;
            if (!(c0 || c1 || c2 || c3)) break;
            const float v = c0 ? d0 : c1 ? d1 : c2 ? d2 : d3;
            if (c0) d0 = INFINITY;
            else if (c1) d1 = INFINITY;
            else if (c2) d2 = INFINITY;
            else d3 = INFINITY;
            set.replace(v, thr);
            thr = set.largest();
        }
        lim = win_upto(stop_r2(thr));
    }
    if (!(thr < INFINITY)) {  // fewer than k + 1 points in the whole window
        defer_query(h, deferred, md_out, i);
        return;
    }
    // every window offset not visited is at least as long as offset o
    const float rbreak = o < WN ? fminf(sqrtf((float)win_len2(o)), (float)(WR + 1)) : (float)(WR + 1);
    const float kth = thr;
    // certificate: every window pixel not visited is at least rbreak away, and
    // every pixel outside the window at least WR + 1
    const float rk = sqrtf(kth), ro = (float)(WR + 1);
    const bool ok = C * rbreak / (an + rbreak) - dev > rk && C * ro / (an + ro) - dev_out > rk;
    if (!ok) {
        // the set holds k + 1 distances of cloud points (the query's own 0
        // among them): its largest bounds the (k + 1)-th smallest from above
        defer_query_bound(h, deferred, md_out, bound, i, kth);
        return;
    }
    const int e = root_exponent(kth);
    const float sc = root_scale(e);
    unsigned sum = 0;
#pragma unroll
    for (int g = 0; g < G; g++) {
        sum += root_fixed(set.top[g], sc);
        const float4 v = set.S[g * WT_T];
        sum += root_fixed(v.x, sc) + root_fixed(v.y, sc) + root_fixed(v.z, sc) + root_fixed(v.w, sc);
    }
    md_out[i] = fixed_mean(sum, e, k);
}

// the window pass's kernel by number of groups, 1 to 13
template <int... g>
auto sor_window_of(int groups, std::integer_sequence<int, g...>) {
    static constexpr decltype(&sor_window_kernel<1>) k[] = {sor_window_kernel<g + 1>...};
    return k[groups - 1];
}

constexpr int FW_CAP = 256;  // tree search: list entries per warp (8 per lane)
constexpr int TS_QUEUE = 256;  // tree search: queued leaves per warp
constexpr int TS_NODES = 2;  // tree search: nodes whose leaves are tested together
constexpr int TS_LEAVES = 2;  // tree search: leaves read together (at most 128 new entries)
constexpr int TS_AROUND = 7;  // tree search: leaves on either side of the query's own that bound it
static_assert((2 * TS_AROUND + 1) * (2 * TS_AROUND + 1) <= FW_CAP && FW_CAP <= TS_QUEUE, "lists of the leaves around");

// Smallest list value v with at least K entries <= v (entries: lane j holds
// keys[r], 0xffffffff = empty; keys are non-negative float bits).  Bisection on
// the bits that stops at the first split with exactly K entries below it: about
// as many steps as the entries have bits, the full 31 only among ties.
__device__ __forceinline__ unsigned warp_kth_key(const unsigned (&keys)[FW_CAP / 32], int K) {
    unsigned lo = 0u, hi = 0x7f800000u;  // +inf bits
    while (lo < hi) {
        const unsigned mid = lo + ((hi - lo) >> 1);
        int c = 0;
#pragma unroll
        for (int r = 0; r < FW_CAP / 32; r++) c += keys[r] <= mid;
        c = __reduce_add_sync(0xffffffffu, c);
        if (c == K) {
            unsigned m = 0u;
#pragma unroll
            for (int r = 0; r < FW_CAP / 32; r++) m = max(m, keys[r] <= mid ? keys[r] : 0u);
            return __reduce_max_sync(0xffffffffu, m);
        }
        if (c > K) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// Tree search: one warp per deferred query.  The warp keeps the squared
// distances below its bound in a list; the bound starts at the window pass's
// (the largest it holds) or, without one, at the nearest farthest corners of
// leaves around the query's own that hold k + 1 points together (7 x 7, then 15 x
// 15; else of the nearest-cornered node and then leaf that holds k + 1), and tightens
// to the (k + 1)-th smallest held whenever the list fills.  With pixel rays the
// bound also limits the search to a rectangle of pixels (the window pass's ray
// bound with the cloud's largest ray distance).  Nodes, then their leaves, then
// the leaves' pixels are read only where the box lies below the bound.  Work is
// handed out through an atomic counter.
//
// Bound by the latency of its dependent loads (one box or pixel access takes
// ~1000 cycles with eight CTAs per SM) and, at the end, by its longest queries
// (5 MP: 47 thousand cycles on average, 230 thousand the longest).  So the leaves
// of two nodes are tested together, a leaf of k + 1 points bounds the search
// before any pixel is read, leaves are queued and read two at a time, and no index
// is divided.  5 MP, k = 30: 105 -> 83 us; 640 x 480, k = 50: 63 -> 22.  Reading four
// or eight leaves at a time or testing four nodes is no faster (a longer list costs
// each selection more).  Where one pixel in ten holds a point no leaf has k + 1, and a
// node's far corner admits a hundred leaves: 1626 x 1236, k = 30, 2.89 ms with the
// nodes' bound alone (the coarse grid 1.57), 1.24 with that of the leaves around.
// The search took the place of a counting-sorted coarse grid with a ring search
// and an occupied-cell search, whose build alone was eleven launches.
__global__ void __launch_bounds__(TS_WARPS * 32) sor_tree_kernel(const float* __restrict__ xyz,
                                                                 const uint8_t* __restrict__ mask, int rows, int cols,
                                                                 int k, int rays, RayParams rp, zl::Tree t,
                                                                 const unsigned* __restrict__ deferred,
                                                                 float* __restrict__ md_out,
                                                                 const float* __restrict__ bound,
                                                                 uint32_t* __restrict__ err) {
    constexpr int NEW = TS_LEAVES * zl::LEAF * zl::LEAF;  // entries a step may add
    static_assert(KNN_MAX_K1 <= FW_CAP - NEW, "a tightened list has room for a step");
    __shared__ float lst[TS_WARPS][FW_CAP];
    __shared__ int2 qpos[TS_WARPS][TS_QUEUE];   // queued leaves: first pixel
    __shared__ float qd2[TS_WARPS][TS_QUEUE];   // and squared box distance
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int K1 = k + 1;
    float* lw = lst[w];
    const unsigned nd = t.head->n_deferred, nwarps = gridDim.x * TS_WARPS;
    // the first query of each warp by its index: thousands of warps asking one
    // counter at once took 4 us
    auto next_item = [&]() {
        unsigned n = 0;
        if (lane == 0) n = nwarps + atomicAdd(&t.head->next, 1u);
        return __shfl_sync(full, n, 0);
    };
    for (unsigned item = blockIdx.x * TS_WARPS + w; item < nd;) {
        const unsigned i = deferred[item];
        const float q[3] = {xyz[3 * (size_t)i], xyz[3 * (size_t)i + 1], xyz[3 * (size_t)i + 2]};
        if (!zl::finite_point(q[0], q[1], q[2])) {  // no neighbours, not even itself
            if (lane == 0) {
                atomicOr(err, 0x10u);
                md_out[i] = 0.f;
            }
            item = next_item();
            continue;
        }
        // entries lie strictly below thr; bounds are met by equality, so they
        // start one float above (finite non-negative floats order as their bits)
        auto above = [](float b) { return b < INFINITY ? __uint_as_float(__float_as_uint(b) + 1u) : INFINITY; };
        const float b0 = bound[i];  // set where md says so
        float thr = INFINITY;
        if (md_out[i] == MD_BOUND) {
            thr = above(b0);
        } else {
            // the farthest corners of the leaves around the query's own that hold k + 1
            // points: the nearest such set, to 2^-7 of its squared distance
            bool bounded = false;
            const int qlx = (int)(i % (unsigned)cols) / zl::LEAF, qly = (int)(i / (unsigned)cols) / zl::LEAF;
            for (int R = 3; R <= TS_AROUND && !bounded; R += TS_AROUND - 3) {
                const int lx0 = max(qlx - R, 0), lx1 = min(qlx + R, t.lw - 1);
                const int ly0 = max(qly - R, 0), ly1 = min(qly + R, t.lh - 1), lnx = lx1 - lx0 + 1;
                const int m = lnx * (ly1 - ly0 + 1);  // at most (2 TS_AROUND + 1)^2
                unsigned held = 0u, hi = 0u, lo = 0u;
                for (int e = lane; e < m; e += 32) {
                    const zl::Box b = zl::load_box(t.leaf, (ly0 + e / lnx) * t.lw + lx0 + e % lnx);
                    const unsigned f = b.n ? __float_as_uint(zl::far_d2(b, q)) : 0x7f800000u;
                    const unsigned c = f < 0x7f800000u ? b.n : 0u;
                    lw[e] = __uint_as_float(f);
                    qpos[w][e].x = (int)c;
                    held += c;
                    hi = max(hi, c ? f : 0u);
                }
                bounded = __reduce_add_sync(full, held) >= (unsigned)K1;
                if (bounded) {
                    hi = __reduce_max_sync(full, hi);
                    while (hi - lo > 0x10000u) {
                        const unsigned mid = lo + ((hi - lo) >> 1);
                        unsigned c = 0u;
                        for (int e = lane; e < m; e += 32) c += __float_as_uint(lw[e]) <= mid ? (unsigned)qpos[w][e].x : 0u;
                        if (__reduce_add_sync(full, c) >= (unsigned)K1) hi = mid;
                        else lo = mid + 1;
                    }
                    thr = above(__uint_as_float(hi));
                }
                __syncwarp();
            }
            if (!bounded) {
                unsigned long long best = ~0ull;  // (distance bits, node)
                for (int n0 = lane; n0 < t.nw * t.nh; n0 += 32) {
                    const zl::Box b = zl::load_box(t.node, n0);
                    if (b.n < (unsigned)K1) continue;
                    const float f = zl::far_d2(b, q);
                    if (f < INFINITY) best = min(best, (unsigned long long)__float_as_uint(f) << 32 | (unsigned)n0);
                }
                for (int off = 16; off; off >>= 1) best = min(best, __shfl_xor_sync(full, best, off));
                if (best != ~0ull) {
                    unsigned fb = (unsigned)(best >> 32);
                    for (int c = lane; c < zl::FAN * zl::FAN; c += 32) {
                        const int l = zl::child_leaf(t, (int)(unsigned)best, c);
                        if (l < 0) continue;
                        const zl::Box b = zl::load_box(t.leaf, l);
                        if (b.n >= (unsigned)K1) fb = min(fb, __float_as_uint(zl::far_d2(b, q)));
                    }
                    thr = above(__uint_as_float(__reduce_min_sync(full, fb)));
                }
            }
        }
        // the nodes of the rectangle of pixels that can hold a point below thr
        int nx0 = 0, ny0 = 0, nx1 = t.nw - 1, ny1 = t.nh - 1;
        if (rays) {
            const int qx = (int)(i % (unsigned)cols), qy = (int)(i / (unsigned)cols);
            float ax, ay, az;
            ray_dir(rp, qx, qy, ax, ay, az);
            const float an = sqrtf(fmaf(ax, ax, fmaf(ay, ay, az * az)));
            const float qn = sqrtf(fmaf(q[0], q[0], fmaf(q[1], q[1], q[2] * q[2])));
            const float C = qn * rp.f / an;
            const float sd = sqrtf(thr) + ray_dev(q[0], q[1], q[2], ax, ay, az) + 2e-5f * qn +
                             __uint_as_float(t.head->ray_dev_bits);
            if (C > sd) {
                const float r = fminf(sd * an / (C - sd) * 1.0001f + 1.f, 1e6f);
                const int ri = (int)r;
                nx0 = max(qx - ri, 0) / zl::NODE;
                ny0 = max(qy - ri, 0) / zl::NODE;
                nx1 = min((qx + ri) / zl::NODE, nx1);
                ny1 = min((qy + ri) / zl::NODE, ny1);
            }
        }
        int n = 0;
        // drops all but the K1 smallest (they are below thr) and tightens thr to the largest of them
        auto tighten = [&]() {
            __syncwarp();
            unsigned keys[FW_CAP / 32];
#pragma unroll
            for (int r = 0; r < FW_CAP / 32; r++) {
                const int e = lane + 32 * r;
                keys[r] = e < n ? __float_as_uint(lw[e]) : 0xffffffffu;
            }
            const unsigned kk = warp_kth_key(keys, K1);
            __syncwarp();
            int m = 0;
#pragma unroll
            for (int r = 0; r < FW_CAP / 32; r++) {
                const bool kp = keys[r] < kk;
                const unsigned bb = __ballot_sync(full, kp);
                if (kp) lw[m + __popc(bb & ((1u << lane) - 1u))] = __uint_as_float(keys[r]);
                m += __popc(bb);
            }
            for (int e = m + lane; e < K1; e += 32) lw[e] = __uint_as_float(kk);  // the ties that fill it
            n = K1;
            thr = __uint_as_float(kk);
            __syncwarp();
        };
        // reads the queued leaves with a box distance below thr
        int nq = 0;
        auto flush = [&]() {
            __syncwarp();
            for (int q0 = 0; q0 < nq; q0 += 32) {
                const float d = q0 + lane < nq ? qd2[w][q0 + lane] : INFINITY;
                for (unsigned m = __ballot_sync(full, d < thr); m; m &= __ballot_sync(full, d < thr)) {
                    float d2[TS_LEAVES][2];
#pragma unroll
                    for (int g = 0; g < TS_LEAVES; g++) {
                        const bool any = m != 0u;
                        const int2 p0 = qpos[w][q0 + (any ? __ffs(m) - 1 : 0)];
                        m &= m - 1;
                        const int px = p0.x + (lane & 7), py = p0.y + (lane >> 3);
                        const bool in0 = any && px < cols && py < rows, in1 = any && px < cols && py + 4 < rows;
                        const size_t j = in0 ? (size_t)py * cols + px : 0, j1 = in1 ? j + 4 * (size_t)cols : 0;
                        const float* a = xyz + 3 * j;
                        const float* b = xyz + 3 * j1;
                        const float ax = __ldg(a), ay = __ldg(a + 1), az = __ldg(a + 2);
                        const float bx = __ldg(b), by = __ldg(b + 1), bz = __ldg(b + 2);
                        const bool v0 = in0 && __ldg(mask + j) != 0, v1 = in1 && __ldg(mask + j1) != 0;
                        d2[g][0] = v0 ? sqdist(ax - q[0], ay - q[1], az - q[2]) : INFINITY;
                        d2[g][1] = v1 ? sqdist(bx - q[0], by - q[1], bz - q[2]) : INFINITY;
                    }
#pragma unroll
                    for (int g = 0; g < TS_LEAVES; g++)
#pragma unroll
                        for (int u = 0; u < 2; u++) {
                            const bool kp = d2[g][u] < thr;  // false for NaN
                            const unsigned bb = __ballot_sync(full, kp);
                            if (kp) lw[n + __popc(bb & ((1u << lane) - 1u))] = d2[g][u];
                            n += __popc(bb);
                        }
                    if (n > FW_CAP - NEW) tighten();
                }
            }
            __syncwarp();
            nq = 0;
        };
        const int rw = nx1 - nx0 + 1, rn = rw * (ny1 - ny0 + 1);
        for (int n0 = 0; n0 < rn; n0 += 32) {
            float nd2 = INFINITY;
            int nx = 0, ny = 0;
            if (n0 + lane < rn) {
                ny = ny0 + (n0 + lane) / rw;
                nx = nx0 + (n0 + lane) % rw;
                const zl::Box b = zl::load_box(t.node, ny * t.nw + nx);
                if (b.n) nd2 = zl::gap_d2(b, q, q);
            }
            for (unsigned nm = __ballot_sync(full, nd2 < thr); nm; nm &= __ballot_sync(full, nd2 < thr)) {
                float ld2[TS_NODES][2];
                int lx[TS_NODES], ly[TS_NODES];
                unsigned fb = 0xffffffffu;
#pragma unroll
                for (int g = 0; g < TS_NODES; g++) {
                    const int nb = nm ? __ffs(nm) - 1 : 0;
                    const bool any = nm != 0u;
                    nm &= nm - 1;
                    lx[g] = __shfl_sync(full, nx, nb) * zl::FAN + (lane & 7);
                    ly[g] = __shfl_sync(full, ny, nb) * zl::FAN + (lane >> 3);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const bool in = any && lx[g] < t.lw && ly[g] + 4 * h < t.lh;
                        const zl::Box b = zl::load_box(t.leaf, in ? (ly[g] + 4 * h) * t.lw + lx[g] : 0);
                        ld2[g][h] = in && b.n ? zl::gap_d2(b, q, q) : INFINITY;
                        if (in && b.n >= (unsigned)K1) fb = min(fb, __float_as_uint(zl::far_d2(b, q)));
                    }
                }
                // a leaf of k + 1 points bounds the search by its farthest corner
                fb = __reduce_min_sync(full, fb);
                if (fb < __float_as_uint(thr)) thr = fminf(thr, above(__uint_as_float(fb)));
#pragma unroll
                for (int g = 0; g < TS_NODES; g++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const bool hit = ld2[g][h] < thr;
                        const unsigned bb = __ballot_sync(full, hit);
                        if (hit) {
                            const int at = nq + __popc(bb & ((1u << lane) - 1u));
                            qpos[w][at] = make_int2(lx[g] * zl::LEAF, (ly[g] + 4 * h) * zl::LEAF);
                            qd2[w][at] = ld2[g][h];
                        }
                        nq += __popc(bb);
                    }
                if (nq > TS_QUEUE - 64 * TS_NODES) flush();
            }
        }
        flush();
        __syncwarp();
        item = next_item();
        if (n < K1) {  // fewer than k + 1 finite points
            if (lane == 0) {
                atomicOr(err, 0x10u);
                md_out[i] = 0.f;
            }
            continue;
        }
        unsigned keys[FW_CAP / 32];
#pragma unroll
        for (int r = 0; r < FW_CAP / 32; r++) {
            const int e = lane + 32 * r;
            keys[r] = e < n ? __float_as_uint(lw[e]) : 0xffffffffu;
        }
        const unsigned kk = warp_kth_key(keys, K1);
        const float kv = __uint_as_float(kk);
        const int ee = root_exponent(kv);
        const float sc = root_scale(ee);
        unsigned part = 0u;
        int below = 0;
#pragma unroll
        for (int r = 0; r < FW_CAP / 32; r++)
            if (keys[r] < kk) {
                part += root_fixed(__uint_as_float(keys[r]), sc);
                below++;
            }
        part = __reduce_add_sync(full, part);
        below = __reduce_add_sync(full, below);
        part += (unsigned)(K1 - below) * root_fixed(kv, sc);
        if (lane == 0) md_out[i] = fixed_mean(part, ee, k);
        __syncwarp();
    }
}

// Sums of the mean distances, a fixed number of blocks striding over the pixels
// (so each thread's share is fixed), the last block to finish adding the block
// partials in block order.  FP64 runs at a small fraction of the FP32 rate: a
// thread's terms add in FP32 with a compensation term (Neumaier: the sum is
// exact to ~2^-24 of its size, like a double sum of these few terms) and go to
// FP64 once.
__device__ __forceinline__ void comp_add(float& sum, float& comp, float x) {
    const float t = sum + x;
    comp += fabsf(sum) >= fabsf(x) ? (sum - t) + x : (x - t) + sum;
    sum = t;
}

constexpr int SOR_STAT_BLOCKS = 456;
constexpr int SOR_STAT_STEPS = 4;

// The sums over a warp of a (in even lanes) and b (in odd lanes): six FP64 adds
// in place of ten (FP64 adds were half of this kernel's time).
__device__ __forceinline__ double warp_sum2(double a, double b) {
    const unsigned full = 0xffffffffu;
    const bool odd = threadIdx.x & 1;
    const double other = __shfl_xor_sync(full, odd ? a : b, 1);
    double v = (odd ? b : a) + other;
#pragma unroll
    for (int off = 2; off < 32; off <<= 1) v += __shfl_xor_sync(full, v, off);
    return v;
}

// Three blocks per SM, four pixels per thread and step and four steps' loads in
// flight; vec: md 16-byte and mask 4-byte aligned, one load each for the four (else
// one per pixel: the same pixels in the same order, so the sums do not depend on
// where the buffers lie).  The
// threshold mean + std_mul * stddev; the classifier compares the float mean
// distances with thr_f, the largest float <= thr, which decides exactly as
// (double)md > thr.
__global__ void __launch_bounds__(GB) sor_stats_kernel(const uint8_t* __restrict__ mask, const float* __restrict__ md,
                                                       size_t n, int vec, int k, double std_mul, zl::Head* h,
                                                       double* __restrict__ part, GridStats* __restrict__ s,
                                                       GridStats* __restrict__ snapshot) {
    float as = 0.f, ac = 0.f, bs = 0.f, bc = 0.f;
    auto take = [&](uint8_t m, float v) {
        if (!m) return;
        comp_add(as, ac, v);
        comp_add(bs, bc, v * v);  // PCL: float square, double sum
    };
    const size_t step = (size_t)gridDim.x * GB, full4 = n / 4;
    size_t g = (size_t)blockIdx.x * GB + threadIdx.x;
    for (; g < full4; g += SOR_STAT_STEPS * step) {
        uchar4 m[SOR_STAT_STEPS];
        float4 v[SOR_STAT_STEPS];
#pragma unroll
        for (int u = 0; u < SOR_STAT_STEPS; u++) {
            m[u] = make_uchar4(0, 0, 0, 0);
            v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            const size_t e = g + u * step;
            if (e >= full4) continue;
            if (vec) {
                m[u] = __ldg(reinterpret_cast<const uchar4*>(mask) + e);
                v[u] = __ldg(reinterpret_cast<const float4*>(md) + e);
            } else {
                m[u] = make_uchar4(mask[4 * e], mask[4 * e + 1], mask[4 * e + 2], mask[4 * e + 3]);
                v[u] = make_float4(md[4 * e], md[4 * e + 1], md[4 * e + 2], md[4 * e + 3]);
            }
        }
#pragma unroll
        for (int u = 0; u < SOR_STAT_STEPS; u++) {
            take(m[u].x, v[u].x); take(m[u].y, v[u].y); take(m[u].z, v[u].z); take(m[u].w, v[u].w);
        }
    }
    for (size_t i = 4 * full4 + (size_t)blockIdx.x * GB + threadIdx.x; i < n; i += step) take(mask[i], md[i]);
    __shared__ double s_sum[GB / 32][2];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // a in lane 0, b in lane 1
    auto block_sum2 = [&](double a, double b) {
        const double v = warp_sum2(a, b);
        if (lane < 2) s_sum[w][lane] = v;
        __syncthreads();
        double r = 0.0;
        if (threadIdx.x < 2)
            for (int j = 0; j < GB / 32; j++) r += s_sum[j][threadIdx.x];
        __syncthreads();
        return r;
    };
    const double mine = block_sum2((double)as + (double)ac, (double)bs + (double)bc);
    if (threadIdx.x < 2) {
        part[2 * blockIdx.x + threadIdx.x] = mine;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&h->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += GB) {
        a += __ldcg(part + 2 * i);
        b += __ldcg(part + 2 * i + 1);
    }
    a = block_sum2(a, b);
    b = __shfl_down_sync(0xffffffffu, a, 1);
    if (threadIdx.x == 0) {
        GridStats o{};
        const double nv = (double)h->n_valid;
        o.n_valid = nv;
        o.md_sum = a;
        o.md_sq = b;
        o.n_deferred = h->n_deferred;
        o.keep_all = nv <= k;  // too few points for a k-neighbourhood: nothing is removed
        if (!o.keep_all) {
            const double mean = a / nv;
            const double var = (b - a * a / nv) / (nv - 1);
            o.thr = mean + std_mul * sqrt(var);
            o.thr_f = __double2float_rd(o.thr);
        }
        *s = o;
        *snapshot = o;
    }
}

// Four pixels per thread; vec: every pointer aligned for vector access.
__global__ void __launch_bounds__(GB) sor_classify_kernel(const float* __restrict__ xyz,
                                                          const uint8_t* __restrict__ mask, size_t n, int vec,
                                                          const GridStats* __restrict__ s,
                                                          const float* __restrict__ md, uint8_t* __restrict__ mask_out,
                                                          float* __restrict__ xyz_out) {
    const size_t g = (size_t)blockIdx.x * GB + threadIdx.x;
    if (4 * g >= n) return;
    const bool all = s->keep_all;
    const float thr = s->thr_f;
    auto keep = [&](uint8_t m, float v) { return m && (all || !(v > thr)); };
    if (vec && 4 * g + 4 <= n) {
        const uchar4 m = __ldg(reinterpret_cast<const uchar4*>(mask) + g);
        const float4 v = __ldg(reinterpret_cast<const float4*>(md) + g);
        float4 p[3];
        if (xyz_out)
#pragma unroll
            for (int c = 0; c < 3; c++) p[c] = __ldg(reinterpret_cast<const float4*>(xyz) + 3 * g + c);
        const bool k0 = keep(m.x, v.x), k1 = keep(m.y, v.y), k2 = keep(m.z, v.z), k3 = keep(m.w, v.w);
        reinterpret_cast<uchar4*>(mask_out)[g] = make_uchar4(k0, k1, k2, k3);
        if (xyz_out) {
            float4* o = reinterpret_cast<float4*>(xyz_out) + 3 * g;
            o[0] = make_float4(k0 ? p[0].x : 0.f, k0 ? p[0].y : 0.f, k0 ? p[0].z : 0.f, k1 ? p[0].w : 0.f);
            o[1] = make_float4(k1 ? p[1].x : 0.f, k1 ? p[1].y : 0.f, k2 ? p[1].z : 0.f, k2 ? p[1].w : 0.f);
            o[2] = make_float4(k2 ? p[2].x : 0.f, k3 ? p[2].y : 0.f, k3 ? p[2].z : 0.f, k3 ? p[2].w : 0.f);
        }
        return;
    }
    for (size_t i = 4 * g; i < n && i < 4 * g + 4; i++) {
        const bool kp = keep(mask[i], md[i]);
        mask_out[i] = kp ? 1 : 0;
        if (xyz_out)
            for (int c = 0; c < 3; c++) xyz_out[3 * i + c] = kp ? xyz[3 * i + c] : 0.f;
    }
}

// ------------------------------------------------------ metric Gaussian ----
//
// out = p + sum w (q - p) / sum w over the points within r = 3 sigma of p.

// The window fast path: the points within r of a query, summed row by row over
// the disk of its window out to the pixel distance beyond which the ray bound
// puts every point farther than r (see sor_window_kernel).  The queries it
// cannot certify are left to metric_gaussian_tree_kernel: a list of (word, its set
// bits), a word being a warp's 16 x 2 pixels.
constexpr int WRG = WR;
constexpr int GW = WT_X + 2 * WRG, GH = WT_Y + 2 * WRG;

// Appends this warp's word of the tile to the list if any bit is set.
__device__ __forceinline__ void list_word(uint2* __restrict__ list, zl::Head* h, unsigned tile, int tid, unsigned word) {
    if ((tid & 31) == 0 && word)
        list[atomicAdd(&h->n_deferred, 1u)] = make_uint2(tile * (WT_T / 32) + (tid >> 5), word);
}

// Without pixel rays every valid point is listed; the others pass through.
__global__ void __launch_bounds__(WT_T) mg_list_kernel(const float* __restrict__ xyz, const uint8_t* __restrict__ mask,
                                                       int rows, int cols, unsigned tiles_x, zl::Tree t,
                                                       uint2* __restrict__ list, float* __restrict__ out) {
    const int tid = threadIdx.x;
    const int x = (int)(blockIdx.x % tiles_x) * WT_X + tid % WT_X, y = (int)(blockIdx.x / tiles_x) * WT_Y + tid / WT_X;
    const bool in = x < cols && y < rows;
    const size_t i = in ? (size_t)y * cols + x : 0;
    const bool left = in && mask[i];
    list_word(list, t.head, blockIdx.x, tid, __ballot_sync(0xffffffffu, left));
    if (in && !left)
        for (int a = 0; a < 3; a++) out[3 * i + a] = xyz[3 * i + a];
}

__global__ void __launch_bounds__(WT_T) mg_window_kernel(const float* __restrict__ xyz,
                                                           const uint8_t* __restrict__ mask, int rows, int cols,
                                                           float r, float inv2s2, RayParams rp,
                                                           zl::Tree t, uint2* __restrict__ list,
                                                           float* __restrict__ out) {
    __shared__ float4 W[GW * GH];
    const int tid = threadIdx.x;
    const int x0 = blockIdx.x * WT_X, y0 = blockIdx.y * WT_Y;
#pragma unroll
    for (int t = tid; t < GW * GH; t += WT_T) {
        const int wx = x0 - WRG + t % GW, wy = y0 - WRG + t / GW;
        // invalid and off-image pixels are NaN: their distance test fails
        const float nan = __int_as_float(0x7fc00000);
        float4 v = make_float4(nan, nan, nan, 0.f);
        if (wx >= 0 && wx < cols && wy >= 0 && wy < rows) {
            const size_t j = (size_t)wy * cols + wx;
            if (mask[j]) v = make_float4(xyz[3 * j], xyz[3 * j + 1], xyz[3 * j + 2], 1.f);
        }
        W[t] = v;
    }
    // the window's pixels are the 3 x 3 tiles around this one (halo 7 < 8), 6 x 6
    // leaves: their points lie within the largest of those leaves' ray distances
    __shared__ unsigned s_td[2];
    if (tid < 64) {
        const int lx = (int)blockIdx.x * 2 - 2 + tid % 8, ly = (int)blockIdx.y * 2 - 2 + tid / 8;
        unsigned td = 0u;
        if (tid % 8 < 6 && tid / 8 < 6 && lx >= 0 && ly >= 0 && lx < t.lw && ly < t.lh)
            td = __float_as_uint(__ldg(t.leaf + 2 * ((size_t)ly * t.lw + lx) + 1).w);
        td = __reduce_max_sync(0xffffffffu, td);
        if ((tid & 31) == 0) s_td[tid >> 5] = td;
    }
    __syncthreads();
    const int tx = tid % WT_X, ty = tid / WT_X;
    const int x = x0 + tx, y = y0 + ty;
    const bool in = x < cols && y < rows;
    const size_t i = in ? (size_t)y * cols + x : 0;
    const float4 q = W[(ty + WRG) * GW + tx + WRG];
    float ax, ay, az;
    ray_dir(rp, x, y, ax, ay, az);
    const float an = sqrtf(fmaf(ax, ax, fmaf(ay, ay, az * az)));
    const float qn = sqrtf(fmaf(q.x, q.x, fmaf(q.y, q.y, q.z * q.z)));
    const float C = qn * rp.f / an;
    // pixels outside the window: within the largest ray distance of all
    const float dev_q = ray_dev(q.x, q.y, q.z, ax, ay, az) + 1e-5f * qn;
    const float dev = dev_q + __uint_as_float(max(s_td[0], s_td[1]));
    const float dev_out = dev_q + __uint_as_float(t.head->ray_dev_bits);
    // window pixels farther than rs from the query hold no point within r,
    // and neither does any pixel outside the window (at least WRG + 1 away)
    const float sd = r + dev;
    const float rs = C > sd ? sd * an / (C - sd) : INFINITY;
    const float ro = (float)(WRG + 1);
    const bool left = q.w != 0.f && (!(rs < ro) || !(C * ro / (an + ro) - dev_out > r));
    const unsigned word = __ballot_sync(0xffffffffu, left);
    list_word(list, t.head, blockIdx.y * gridDim.x + blockIdx.x, tid, word);
    if (!in || left) return;
    if (q.w == 0.f) {  // invalid points pass through
        out[3 * i] = xyz[3 * i];
        out[3 * i + 1] = xyz[3 * i + 1];
        out[3 * i + 2] = xyz[3 * i + 2];
        return;
    }
    const float r2 = r * r;
    const int wc = (ty + WRG) * GW + tx + WRG;
    // The disk of pixels within rs, row by row (the query itself included:
    // offset 0, weight exactly 1); w = 2^(d2 kq), kq = -log2(e) / (2 s^2)
    const float kq = -1.44269504088896341f * inv2s2;
    float sx = 0.f, sy = 0.f, sz = 0.f, sw = 0.f;
    const int R2 = (int)(rs * rs);  // offsets with dx^2 + dy^2 <= R2 (< (WRG + 1)^2)
    const int R = min((int)rs, WRG);
#pragma unroll 1
    for (int dy = -R; dy <= R; dy++) {
        // exact floor of the root: a root of a non-square below 64 lies at least
        // 0.06 from an integer, and the approximate root's error is far smaller
        const int w = min((int)(root_approx((float)max(R2 - dy * dy, 0)) + 0.03f), WRG);
        const float4* row = W + wc + dy * GW;
#pragma unroll 2
        for (int dx = -w; dx <= w; dx++) {
            const float4 p = row[dx];
            const float ex = p.x - q.x, ey = p.y - q.y, ez = p.z - q.z;
            const float d2 = sqdist(ex, ey, ez);
            if (!(d2 <= r2)) continue;  // also every invalid pixel (NaN)
            float wt;
            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(wt) : "f"(d2 * kq));
            sx = fmaf(wt, ex, sx); sy = fmaf(wt, ey, sy); sz = fmaf(wt, ez, sz);
            sw += wt;
        }
    }
    const float iw = 1.0f / sw;
    out[3 * i] = q.x + sx * iw;
    out[3 * i + 1] = q.y + sy * iw;
    out[3 * i + 2] = q.z + sz * iw;
}

// Queries over the tree's leaves, a warp per listed word of 16 x 2 pixels: the box of
// the warp's queries picks the leaves and their points within r of it, which go through
// shared memory, each lane summing those within r of its own query.  64-bit fixed-point
// sums (each term rounded on its own): the result depends neither on the visiting order
// nor on the list's.  When nothing is listed, the launch costs one wave of blocks that
// return at once (the hash grid it replaced took ten gated launches: 102 -> 63 us for
// a 1280 x 1024 cloud).  With every query left to it (no pixel rays) a 2448 x 2048
// cloud takes 6.1 ms at sigma 0.5 and 14 ms at 1, against 10 and 29 ms with the grid.
//
// A cloud after the pixel Gaussian has its rejected pixels valid at the origin, all
// within r of each other, and most of them on the image's border: a few lanes of some
// words with thousands of neighbours.  So the words are listed, which spreads them over
// the SMs (strided, the border tiles of a 1024-pixel image fall to one block in 64), and
// only the points near the queries' box are summed over, not a leaf's 64 pixels: such a
// 1024 x 768 cloud 9.2 -> 2.7 ms (the grid: 5.7).
constexpr int MT_WARPS = 8;
__global__ void __launch_bounds__(MT_WARPS * 32) metric_gaussian_tree_kernel(
    const float* __restrict__ xyz, const uint8_t* __restrict__ mask, int rows, int cols, float r2, float inv2s2,
    zl::Tree t, const uint2* __restrict__ list, float* __restrict__ out) {
    const unsigned words = t.head->n_deferred;
    __shared__ float4 pts[MT_WARPS][zl::LEAF * zl::LEAF];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float4* pw = pts[w];
    const unsigned tiles_x = (cols + WT_X - 1) / WT_X;
    const int nn = t.nw * t.nh;
    const float r = sqrtf(r2), sc = 1099511627776.0f / r;  // 2^40 / r
    for (unsigned item = blockIdx.x * MT_WARPS + w; item < words; item += gridDim.x * MT_WARPS) {
        const uint2 e = list[item];
        const unsigned tile = e.x / (WT_T / 32);
        const int x = (int)(tile % tiles_x) * WT_X + (lane & 15);
        const int y = (int)(tile / tiles_x) * WT_Y + (int)(e.x % (WT_T / 32)) * 2 + (lane >> 4);
        const bool act = e.y >> lane & 1u;
        const size_t i = act ? (size_t)y * cols + x : 0;
        float q[3] = {0.f, 0.f, 0.f}, lo[3], hi[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            if (act) q[a] = xyz[3 * i + a];
            const unsigned key = zl::fkey(q[a]);
            lo[a] = zl::keyf(__reduce_min_sync(full, act ? key : ~0u));
            hi[a] = zl::keyf(__reduce_max_sync(full, act ? key : 0u));
        }
        long long sx = 0, sy = 0, sz = 0, sw = 0;
        for (int n0 = 0; n0 < nn; n0 += 32) {
            bool hit = false;
            if (n0 + lane < nn) {
                const zl::Box b = zl::load_box(t.node, n0 + lane);
                hit = b.n && zl::gap_d2(b, lo, hi) <= r2;
            }
            for (unsigned nm = __ballot_sync(full, hit); nm; nm &= nm - 1) {
                const int nb = n0 + __ffs(nm) - 1;
#pragma unroll 1
                for (int h = 0; h < 2; h++) {
                    const int ll = zl::child_leaf(t, nb, lane + 32 * h);
                    bool lhit = false;
                    if (ll >= 0) {
                        const zl::Box b = zl::load_box(t.leaf, ll);
                        lhit = b.n && zl::gap_d2(b, lo, hi) <= r2;
                    }
                    for (unsigned lm = __ballot_sync(full, lhit); lm; lm &= lm - 1) {
                        const int l = __shfl_sync(full, ll, __ffs(lm) - 1);
                        const int px = (l % t.lw) * zl::LEAF + (lane & 7), py = (l / t.lw) * zl::LEAF + (lane >> 3);
                        // the leaf's points within r of the queries' box
                        int np = 0;
                        __syncwarp();
#pragma unroll
                        for (int u = 0; u < 2; u++) {
                            const bool in = px < cols && py + 4 * u < rows;
                            const size_t j = in ? (size_t)(py + 4 * u) * cols + px : 0;
                            const float vx = __ldg(xyz + 3 * j), vy = __ldg(xyz + 3 * j + 1), vz = __ldg(xyz + 3 * j + 2);
                            const bool v = in && __ldg(mask + j) != 0 &&
                                           zl::gap_d2(zl::Box{{vx, vy, vz}, {vx, vy, vz}, 1u}, lo, hi) <= r2;
                            const unsigned bb = __ballot_sync(full, v);
                            if (v) pw[np + __popc(bb & ((1u << lane) - 1u))] = make_float4(vx, vy, vz, 0.f);
                            np += __popc(bb);
                        }
                        __syncwarp();
                        if (act)
#pragma unroll 4
                            for (int k = 0; k < np; k++) {
                                const float4 p = pw[k];
                                const float dx = p.x - q[0], dy = p.y - q[1], dz = p.z - q[2];
                                const float d2 = sqdist(dx, dy, dz);
                                if (!(d2 <= r2)) continue;
                                const float g = __expf(-d2 * inv2s2);
                                sx += __float2ll_rn(g * dx * sc);
                                sy += __float2ll_rn(g * dy * sc);
                                sz += __float2ll_rn(g * dz * sc);
                                sw += __float2ll_rn(g * 1099511627776.0f);
                            }
                    }
                }
            }
        }
        if (act) {
            // (S / 2^40 * r) / (W / 2^40); W = 0 for a point without finite coordinates,
            // which is nobody's neighbour, not its own either: it stays
            const double kd = sw ? (double)r / (double)sw : 0.0;
            out[3 * i] = (float)((double)q[0] + (double)sx * kd);
            out[3 * i + 1] = (float)((double)q[1] + (double)sy * kd);
            out[3 * i + 2] = (float)((double)q[2] + (double)sz * kd);
        }
    }
}

unsigned table_size(size_t want) {
    unsigned t = 1024;
    while (t < want && t < (1u << 30)) t <<= 1;
    return t;
}

// The tile search's grid: about 4 points per bucket.
struct GridScratch {
    unsigned tsize;
    uint2* tab;
    float4* pts;
    unsigned* counts;
    unsigned* tot;
    double* part;  // block partials of the spacing passes (2 per block)
};

size_t grid_bytes(size_t n) {
    const unsigned t = table_size(n / 4);
    return zim_align256((size_t)t * 8) + zim_align256(n * 16) + zim_align256((size_t)t * 4) +
           zim_align256(((t + SCAN_B - 1) / SCAN_B) * 4) + zim_align256((size_t)SPACING_BLOCKS * 2 * sizeof(double));
}

zim_status carve_grid(zim_ctx* ctx, size_t n, GridScratch& G) {
    G.tsize = table_size(n / 4);
    G.tab = (uint2*)zim_scratch_take(ctx, (size_t)G.tsize * 8);
    G.pts = (float4*)zim_scratch_take(ctx, n * 16);
    G.counts = (unsigned*)zim_scratch_take(ctx, (size_t)G.tsize * 4);
    G.tot = (unsigned*)zim_scratch_take(ctx, ((G.tsize + SCAN_B - 1) / SCAN_B) * 4);
    G.part = (double*)zim_scratch_take(ctx, (size_t)SPACING_BLOCKS * 2 * sizeof(double));
    if (!G.tab || !G.pts || !G.counts || !G.tot || !G.part)
        return zim_fail(ctx, ZIM_ERR_OUT_OF_MEMORY, "grid scratch carve");
    return ZIM_OK;
}

// The grid's cell size, then its table (counting sort of the points by slot).
zim_status build_grid(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows, int cols, float factor,
                      GridStats* stats, GridScratch& G, cudaStream_t st) {
    const size_t n = (size_t)rows * cols;
    const unsigned sblk = (unsigned)std::min<size_t>((n + GB - 1) / GB, SPACING_BLOCKS);
    stats_init_kernel<<<1, 1, 0, st>>>(stats);
    spacing1_kernel<<<sblk, GB, 0, st>>>(xyz, mask, rows, cols, stats, G.part);
    spacing_total_kernel<<<1, SPACING_BLOCKS, 0, st>>>(G.part, (int)sblk, 1, stats);
    spacing2_kernel<<<sblk, GB, 0, st>>>(xyz, mask, rows, cols, stats, G.part);
    spacing_total_kernel<<<1, SPACING_BLOCKS, 0, st>>>(G.part, (int)sblk, 2, stats);
    cell_kernel<<<1, 1, 0, st>>>(stats, factor);
    // grids sized to the GPU (the kernels stride): 8 blocks of 256 per SM,
    // 2 of the scans' 1024
    const unsigned sms = (unsigned)(ctx->sm_count > 0 ? ctx->sm_count : 152);
    const unsigned nblk = (unsigned)std::min<size_t>((n + GB - 1) / GB, 8 * sms);
    const unsigned T = G.tsize, nb = (T + SCAN_B - 1) / SCAN_B;
    const unsigned tblk = std::min((T + GB - 1) / GB, 8 * sms), cblk = std::min(nb, 2 * sms);
    zero_kernel<<<tblk, GB, 0, st>>>(G.counts, T);
    hash_count_kernel<<<nblk, GB, 0, st>>>(xyz, mask, n, stats, T - 1, G.counts);
    scan_blocks_kernel<<<cblk, SCAN_B, 0, st>>>(G.counts, G.tab, T, G.tot);
    scan_totals_kernel<<<1, SCAN_B, 0, st>>>(G.tot, (int)nb);
    scan_add_kernel<<<cblk, SCAN_B, 0, st>>>(G.tab, T, G.tot);
    zero_kernel<<<tblk, GB, 0, st>>>(G.counts, T);
    hash_scatter_kernel<<<nblk, GB, 0, st>>>(xyz, mask, n, stats, T - 1, G.tab, G.counts, G.pts);
    ctx->launches += 13;
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}

// Words of the metric Gaussian's list.
size_t mg_words(int rows, int cols) {
    return (size_t)((cols + WT_X - 1) / WT_X) * ((rows + WT_Y - 1) / WT_Y) * (WT_T / 32);
}

}  // namespace

// Scratch of the filters of one cloud (they carve it in turn): SOR's statistics,
// mean distances, deferred queries and bounds, the tree, and without pixel rays
// the grid; the metric Gaussian needs less (the tree and its list).
size_t zim_grid_scratch_bytes(int rows, int cols, bool rays) {
    const size_t n = (size_t)rows * cols;
    return zim_leaf_bytes(rows, cols) + zim_align256(sizeof(GridStats)) + 3 * zim_align256(n * 4) +
           zim_align256((size_t)SOR_STAT_BLOCKS * 2 * sizeof(double)) + (rays ? 0 : grid_bytes(n)) +
           zim_align256(mg_words(rows, cols) * sizeof(uint2));
}

zim_status zim_sor_launch(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows, int cols, int mean_k,
                          double std_mul, float* xyz_out, uint8_t* mask_out, float* mean_dist,
                          const zim_ray_model& rays, cudaStream_t st) {
    const size_t n = (size_t)rows * cols;
    zl::Tree t;
    zim_status s = zim_leaf_carve(ctx, rows, cols, t);
    if (s) return s;
    GridStats* stats = (GridStats*)zim_scratch_take(ctx, sizeof(GridStats));
    float* md = mean_dist ? mean_dist : (float*)zim_scratch_take(ctx, n * 4);
    unsigned* deferred = (unsigned*)zim_scratch_take(ctx, n * 4);
    float* bound = (float*)zim_scratch_take(ctx, n * 4);  // per pixel: a deferred query's bound (md = MD_BOUND)
    double* part = (double*)zim_scratch_take(ctx, (size_t)SOR_STAT_BLOCKS * 2 * sizeof(double));
    if (!stats || !md || !deferred || !bound || !part) return zim_fail(ctx, ZIM_ERR_OUT_OF_MEMORY, "SOR scratch carve");
    const RayParams rp = zt::ray_params(rays);
    s = zim_leaf_build(ctx, xyz, mask, rows, cols, rays.valid ? &rp : nullptr, t, st);
    if (s) return s;
    if (rays.valid) {
        const dim3 wgrid((cols + WT_X - 1) / WT_X, (rows + WT_Y - 1) / WT_Y);
        const int groups = (mean_k + NS_N) / NS_N;  // (k + 1) / NS_N rounded up
        const size_t wsm = WIN_BYTES + sizeof(float4) * groups * WT_T;
        auto kern = sor_window_of(groups, std::make_integer_sequence<int, (KNN_MAX_K1 + NS_N - 1) / NS_N>{});
        ZIM_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wsm));
        kern<<<wgrid, WT_T, wsm, st>>>(xyz, mask, rows, cols, mean_k, rp, t, md, deferred, bound);
    } else {
        // cell ~ 3.5 x spacing: the (k+1)-th neighbour of a surface point
        // lies within one ring for ~98% of points at k = 30
        const float factor = 3.5f * sqrtf(fmaxf(1.0f, (float)mean_k / 30.0f));
        GridScratch G;
        s = carve_grid(ctx, n, G);
        if (s) return s;
        s = build_grid(ctx, xyz, mask, rows, cols, factor, stats, G, st);
        if (s) return s;
        const dim3 tgrid((cols + TILE_X - 1) / TILE_X, (rows + TILE_Y - 1) / TILE_Y);
        const size_t tsm = (size_t)TILE_MAX_CAND * sizeof(float4);
        // dynamic + static shared memory exceeds the default 48 KB (attribute is per device: set it every call)
        ZIM_CUDA_TRY(ctx, cudaFuncSetAttribute(sor_knn_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsm));
        sor_knn_tile_kernel<<<tgrid, TILE_T, tsm, st>>>(xyz, mask, rows, cols, mean_k, Level{G.tab, G.pts, G.tsize - 1},
                                                        stats, t.head, md, deferred);
    }
    const unsigned sms = (unsigned)(ctx->sm_count > 0 ? ctx->sm_count : 152);
    sor_tree_kernel<<<8 * sms, TS_WARPS * 32, 0, st>>>(xyz, mask, rows, cols, mean_k, rays.valid, rp, t, deferred,
                                                       md, bound, ctx->d_error);
    const size_t quads = (n + 3) / 4;
    const uintptr_t mal = (uintptr_t)mask | (uintptr_t)mask_out;
    const int vs = ((uintptr_t)md & 15) == 0 && ((uintptr_t)mask & 3) == 0;
    const int vc = vs && (mal & 3) == 0 && (((uintptr_t)xyz | (uintptr_t)xyz_out) & 15) == 0;
    const unsigned pblk = (unsigned)std::min<size_t>((quads + GB - 1) / GB, SOR_STAT_BLOCKS);
    static_assert(sizeof(GridStats) <= 256, "stats snapshot buffer");
    sor_stats_kernel<<<pblk, GB, 0, st>>>(mask, md, n, vs, mean_k, std_mul, t.head, part, stats,
                                          (GridStats*)ctx->d_sor_stats);
    sor_classify_kernel<<<(unsigned)((quads + GB - 1) / GB), GB, 0, st>>>(xyz, mask, n, vc, stats, md, mask_out, xyz_out);
    ctx->launches += 4;
    ctx->have_sor_stats = true;
    ctx->last_sor_std_mul = std_mul;
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}

zim_status zim_metric_gaussian_launch(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows, int cols,
                                      double sigma, float* out, const zim_ray_model& rays, cudaStream_t st) {
    zl::Tree t;
    zim_status s = zim_leaf_carve(ctx, rows, cols, t);
    if (s) return s;
    const float rad = (float)(3.0 * sigma);
    const RayParams rp = zt::ray_params(rays);
    s = zim_leaf_build(ctx, xyz, mask, rows, cols, rays.valid ? &rp : nullptr, t, st);
    if (s) return s;
    const float inv2s2 = (float)(1.0 / (2.0 * sigma * sigma));
    const size_t words = mg_words(rows, cols);
    uint2* list = (uint2*)zim_scratch_take(ctx, words * sizeof(uint2));
    if (!list) return zim_fail(ctx, ZIM_ERR_OUT_OF_MEMORY, "metric Gaussian scratch carve");
    const dim3 tgrid((cols + WT_X - 1) / WT_X, (rows + WT_Y - 1) / WT_Y);
    if (rays.valid)
        mg_window_kernel<<<tgrid, WT_T, 0, st>>>(xyz, mask, rows, cols, rad, inv2s2, rp, t, list, out);
    else
        mg_list_kernel<<<tgrid.x * tgrid.y, WT_T, 0, st>>>(xyz, mask, rows, cols, tgrid.x, t, list, out);
    const unsigned mblk = (unsigned)std::min<size_t>((words + MT_WARPS - 1) / MT_WARPS,
                                                     8 * (ctx->sm_count > 0 ? ctx->sm_count : 152));
    metric_gaussian_tree_kernel<<<mblk, MT_WARPS * 32, 0, st>>>(xyz, mask, rows, cols, rad * rad, inv2s2, t, list, out);
    ctx->launches += 2;
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}

extern "C" ZIM_API zim_status zim_filter_sor(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows, int cols,
                                             int mean_k, double std_mul, uint8_t* mask_out, float* mean_dist,
                                             void* stream) {
    if (!ctx) return ZIM_ERR_INVALID_ARG;
    if (!xyz || !mask || !mask_out || rows <= 0 || cols <= 0) return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "bad argument");
    if (mean_k < 1 || mean_k + 1 > KNN_MAX_K1) return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "mean_k must be in [1, 63]");
    ZIM_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    // a cloud of the calibrated rectified size: its pixels' rays as the window hint
    const zim_ray_model rays = rows == ctx->rect_h && cols == ctx->rect_w ? zim_rays_of(ctx, true, 0, 0)
                                                                          : zim_ray_model{};
    zim_status s = zim_scratch_reserve(ctx, zim_grid_scratch_bytes(rows, cols, rays.valid != 0));
    if (s) return s;
    zim_scratch_reset(ctx);
    return zim_sor_launch(ctx, xyz, mask, rows, cols, mean_k, std_mul, nullptr, mask_out, mean_dist, rays,
                          zim_stream(stream));
}

extern "C" ZIM_API zim_status zim_filter_sor_stats(zim_ctx* ctx, zim_sor_stats* out) {
    if (!ctx) return ZIM_ERR_INVALID_ARG;
    if (!out || !ctx->have_sor_stats) return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "no SOR run on this context");
    GridStats h;
    ZIM_CUDA_TRY(ctx, cudaDeviceSynchronize());
    ZIM_CUDA_TRY(ctx, cudaMemcpy(&h, ctx->d_sor_stats, sizeof h, cudaMemcpyDeviceToHost));
    const double nv = h.n_valid;
    out->n_valid = nv;
    out->mean = nv > 0 ? h.md_sum / nv : 0.0;
    out->stddev = nv > 1 ? sqrt((h.md_sq - h.md_sum * h.md_sum / nv) / (nv - 1)) : 0.0;
    out->threshold = out->mean + ctx->last_sor_std_mul * out->stddev;
    out->n_far_search = h.n_deferred;
    return ZIM_OK;
}

extern "C" ZIM_API zim_status zim_filter_metric_gaussian(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows,
                                                         int cols, double sigma, float* out, void* stream) {
    if (!ctx) return ZIM_ERR_INVALID_ARG;
    if (!xyz || !mask || !out || rows <= 0 || cols <= 0 || !(sigma > 0))
        return zim_fail(ctx, ZIM_ERR_INVALID_ARG, "bad argument");
    ZIM_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    const zim_ray_model rays = rows == ctx->rect_h && cols == ctx->rect_w ? zim_rays_of(ctx, true, 0, 0)
                                                                          : zim_ray_model{};
    zim_status s = zim_scratch_reserve(ctx, zim_grid_scratch_bytes(rows, cols, rays.valid != 0));
    if (s) return s;
    zim_scratch_reset(ctx);
    return zim_metric_gaussian_launch(ctx, xyz, mask, rows, cols, sigma, out, rays, zim_stream(stream));
}