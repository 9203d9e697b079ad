// leaf.cu -- the bounding-box tree of an organised cloud (zim_leaf.cuh).
#include "zim_leaf.cuh"

namespace {

constexpr int LW = 16, LB = 32 * LW;  // a block per node: 16 warps of four leaves (32 x 8 pixels) each

struct Acc {
    float lo[3], hi[3], dev2;
    unsigned n;
};

__device__ __forceinline__ void merge_lane(Acc& a, int off) {
    const unsigned full = 0xffffffffu;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        a.lo[c] = fminf(a.lo[c], __shfl_xor_sync(full, a.lo[c], off));
        a.hi[c] = fmaxf(a.hi[c], __shfl_xor_sync(full, a.hi[c], off));
    }
    a.dev2 = fmaxf(a.dev2, __shfl_xor_sync(full, a.dev2, off));
    a.n += __shfl_xor_sync(full, a.n, off);
}

__device__ __forceinline__ void store_box(float4* boxes, int i, const Acc& a) {
    boxes[2 * (size_t)i] = make_float4(a.lo[0], a.lo[1], a.lo[2], __uint_as_float(a.n));
    boxes[2 * (size_t)i + 1] = make_float4(a.hi[0], a.hi[1], a.hi[2], sqrtf(a.dev2));
}

// One pass over the cloud, 13 B per pixel read and 0.5 B written.  A lane takes a
// column of eight pixels, so a leaf's box is eight in-register steps and three
// shuffles; a warp per leaf with a reduction per coordinate took 2.3 times the
// instructions.  The ray distance is compared squared (zt::ray_dev's value, one
// root per box).
__global__ void __launch_bounds__(LB) leaf_kernel(const float* __restrict__ xyz, const uint8_t* __restrict__ mask,
                                                  int rows, int cols, int rays, zt::RayParams rp, zl::Tree t) {
    __shared__ Acc s_leaf[zl::FAN * zl::FAN];
    __shared__ unsigned s_valid[LW];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nx = (int)(blockIdx.x % (unsigned)t.nw), ny = (int)(blockIdx.x / (unsigned)t.nw);
    const int x = nx * zl::NODE + (w & 1) * 32 + lane, y0 = ny * zl::NODE + (w >> 1) * zl::LEAF;
    Acc a{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}, 0.f, 0u};
    unsigned nv = 0u;
#pragma unroll
    for (int h = 0; h < zl::LEAF; h += 4) {
        float p[4][3];
        bool v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int y = y0 + h + u;
            const bool in = x < cols && y < rows;
            const size_t i = in ? (size_t)y * cols + x : 0;
            v[u] = in && __ldg(mask + i) != 0;
#pragma unroll
            for (int c = 0; c < 3; c++) p[u][c] = __ldg(xyz + 3 * i + c);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (!v[u]) continue;
            nv++;
            if (zl::finite_point(p[u][0], p[u][1], p[u][2])) {
                a.n++;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    a.lo[c] = fminf(a.lo[c], p[u][c]);
                    a.hi[c] = fmaxf(a.hi[c], p[u][c]);
                }
            }
            if (rays) {
                float ax, ay, az;
                zt::ray_dir(rp, x, y0 + h + u, ax, ay, az);
                const float cx = fmaf(p[u][1], az, -p[u][2] * ay), cy = fmaf(p[u][2], ax, -p[u][0] * az),
                            cz = fmaf(p[u][0], ay, -p[u][1] * ax);
                const float d2 = __fdividef(fmaf(cx, cx, fmaf(cy, cy, cz * cz)), fmaf(ax, ax, fmaf(ay, ay, az * az)));
                a.dev2 = fmaxf(a.dev2, d2 == d2 ? d2 : INFINITY);  // NaN counts as unbounded
            }
        }
    }
#pragma unroll
    for (int off = 4; off; off >>= 1) merge_lane(a, off);
    const int lx = x / zl::LEAF, ly = y0 / zl::LEAF;
    if ((lane & 7) == 0) {
        s_leaf[w * 4 + (lane >> 3)] = a;
        if (lx < t.lw && ly < t.lh) store_box(t.leaf, ly * t.lw + lx, a);
    }
    nv = __reduce_add_sync(0xffffffffu, nv);
    if (lane == 0) s_valid[w] = nv;
    __syncthreads();
    if (w) return;
    a = s_leaf[lane];
    const Acc b = s_leaf[lane + 32];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        a.lo[c] = fminf(a.lo[c], b.lo[c]);
        a.hi[c] = fmaxf(a.hi[c], b.hi[c]);
    }
    a.dev2 = fmaxf(a.dev2, b.dev2);
    a.n += b.n;
#pragma unroll
    for (int off = 16; off; off >>= 1) merge_lane(a, off);
    nv = __reduce_add_sync(0xffffffffu, lane < LW ? s_valid[lane] : 0u);
    if (lane == 0) {
        store_box(t.node, blockIdx.x, a);
        if (nv) atomicAdd(&t.head->n_valid, nv);
        if (a.dev2 > 0.f) atomicMax(&t.head->ray_dev_bits, __float_as_uint(sqrtf(a.dev2)));
    }
}

struct Dims {
    int lw, lh, nw, nh;
    size_t node, leaf;
};

Dims dims(int rows, int cols) {
    Dims d;
    d.lw = (cols + zl::LEAF - 1) / zl::LEAF;
    d.lh = (rows + zl::LEAF - 1) / zl::LEAF;
    d.nw = (d.lw + zl::FAN - 1) / zl::FAN;
    d.nh = (d.lh + zl::FAN - 1) / zl::FAN;
    d.node = (size_t)d.nw * d.nh * 2 * sizeof(float4);
    d.leaf = (size_t)d.lw * d.lh * 2 * sizeof(float4);
    return d;
}

}  // namespace

size_t zim_leaf_bytes(int rows, int cols) {
    const Dims d = dims(rows, cols);
    return zim_align256(sizeof(zl::Head)) + zim_align256(d.node) + zim_align256(d.leaf);
}

zim_status zim_leaf_carve(zim_ctx* ctx, int rows, int cols, zl::Tree& t) {
    const Dims d = dims(rows, cols);
    t.head = (zl::Head*)zim_scratch_take(ctx, sizeof(zl::Head));
    t.node = (float4*)zim_scratch_take(ctx, d.node);
    t.leaf = (float4*)zim_scratch_take(ctx, d.leaf);
    if (!t.head || !t.node || !t.leaf) return zim_fail(ctx, ZIM_ERR_OUT_OF_MEMORY, "leaf tree scratch");
    t.lw = d.lw; t.lh = d.lh; t.nw = d.nw; t.nh = d.nh;
    return ZIM_OK;
}

zim_status zim_leaf_build(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows, int cols,
                          const zt::RayParams* rays, zl::Tree& t, cudaStream_t st) {
    ZIM_CUDA_TRY(ctx, cudaMemsetAsync(t.head, 0, sizeof(zl::Head), st));
    leaf_kernel<<<(unsigned)t.nw * (unsigned)t.nh, LB, 0, st>>>(xyz, mask, rows, cols, rays ? 1 : 0,
                                                                rays ? *rays : zt::RayParams{}, t);
    ctx->launches += 1;
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}
