// leaf.cu -- the bounding-box tree of an organised cloud (zim_leaf.cuh).
#include "zim_leaf.cuh"

namespace {

constexpr int LB = 32 * zl::FAN;  // a warp per leaf, a row of one node's leaves per block

// One pass over the cloud: 13 B per pixel read, 0.5 B written.  A warp takes a
// leaf (two pixels a lane), so its box is six warp reductions; the eight leaves
// of a block meet in shared memory and go to their node as seven atomics.
__global__ void __launch_bounds__(LB) leaf_kernel(const float* __restrict__ xyz, const uint8_t* __restrict__ mask,
                                                  int rows, int cols, int rays, zt::RayParams rp, zl::Tree t) {
    __shared__ unsigned s_node[zl::NODE_WORDS], s_dev;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x < zl::NODE_WORDS) s_node[threadIdx.x] = 0u;
    if (threadIdx.x == 0) s_dev = 0u;
    __syncthreads();
    const int nx = (int)(blockIdx.x % (unsigned)t.nw), ly = (int)(blockIdx.x / (unsigned)t.nw);
    const int lx = nx * zl::FAN + w;
    const int x = lx * zl::LEAF + (lane & 7), y0 = ly * zl::LEAF + (lane >> 3);
    float p[2][3];
    bool v[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int y = y0 + 4 * u;
        const bool in = x < cols && y < rows;
        const size_t i = in ? (size_t)y * cols + x : 0;
        v[u] = in && __ldg(mask + i) != 0;
#pragma unroll
        for (int a = 0; a < 3; a++) p[u][a] = in ? __ldg(xyz + 3 * i + a) : 0.f;
    }
    unsigned mn[3] = {~0u, ~0u, ~0u}, mx[3] = {0u, 0u, 0u}, dev = 0u;
    unsigned nv = 0u, nf = 0u;
#pragma unroll
    for (int u = 0; u < 2; u++) {
        // points with a NaN or infinite coordinate are nobody's neighbour: outside every box
        const bool f = v[u] && isfinite(p[u][0]) && isfinite(p[u][1]) && isfinite(p[u][2]);
        nv += __popc(__ballot_sync(0xffffffffu, v[u]));
        nf += __popc(__ballot_sync(0xffffffffu, f));
        if (f)
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const unsigned k = zl::fkey(p[u][a]);
                mn[a] = min(mn[a], k);
                mx[a] = max(mx[a], k);
            }
        if (rays && v[u]) {
            float ax, ay, az;
            zt::ray_dir(rp, x, y0 + 4 * u, ax, ay, az);
            const float d = zt::ray_dev(p[u][0], p[u][1], p[u][2], ax, ay, az);
            dev = max(dev, __float_as_uint(d == d ? d : INFINITY));  // NaN counts as unbounded
        }
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        mn[a] = __reduce_min_sync(0xffffffffu, mn[a]);
        mx[a] = __reduce_max_sync(0xffffffffu, mx[a]);
    }
    if (rays) dev = __reduce_max_sync(0xffffffffu, dev);
    if (lane == 0 && lx < t.lw) {
        const size_t l = (size_t)ly * t.lw + lx;
        const float inf = INFINITY;
        t.leaf[2 * l] = nf ? make_float4(zl::keyf(mn[0]), zl::keyf(mn[1]), zl::keyf(mn[2]), __uint_as_float(nf))
                           : make_float4(inf, inf, inf, __uint_as_float(0u));
        t.leaf[2 * l + 1] = nf ? make_float4(zl::keyf(mx[0]), zl::keyf(mx[1]), zl::keyf(mx[2]), __uint_as_float(dev))
                               : make_float4(-inf, -inf, -inf, __uint_as_float(dev));
        if (nf) {
#pragma unroll
            for (int a = 0; a < 3; a++) {
                atomicMax(&s_node[a], ~mn[a]);
                atomicMax(&s_node[3 + a], mx[a]);
            }
            atomicAdd(&s_node[6], nf);
        }
        if (nv) atomicAdd(&s_node[7], nv);
        if (dev) atomicMax(&s_dev, dev);
    }
    __syncthreads();
    unsigned* nd = t.node + (size_t)zl::NODE_WORDS * ((ly / zl::FAN) * t.nw + nx);
    const int j = threadIdx.x;
    if (j < 6 && s_node[j]) atomicMax(nd + j, s_node[j]);
    if (j == 6 && s_node[6]) atomicAdd(nd + 6, s_node[6]);
    if (j == 7 && s_node[7]) atomicAdd(&t.head->n_valid, s_node[7]);
    if (j == 8 && s_dev) atomicMax(&t.head->ray_dev_bits, s_dev);
}

struct Dims {
    int lw, lh, nw, nh;
    size_t zeroed, leaf;
};

Dims dims(int rows, int cols) {
    Dims d;
    d.lw = (cols + zl::LEAF - 1) / zl::LEAF;
    d.lh = (rows + zl::LEAF - 1) / zl::LEAF;
    d.nw = (d.lw + zl::FAN - 1) / zl::FAN;
    d.nh = (d.lh + zl::FAN - 1) / zl::FAN;
    d.zeroed = sizeof(zl::Head) + (size_t)d.nw * d.nh * zl::NODE_WORDS * 4;
    d.leaf = (size_t)d.lw * d.lh * 2 * sizeof(float4);
    return d;
}

}  // namespace

size_t zim_leaf_bytes(int rows, int cols) {
    const Dims d = dims(rows, cols);
    return zim_align256(d.zeroed) + zim_align256(d.leaf);
}

zim_status zim_leaf_carve(zim_ctx* ctx, int rows, int cols, zl::Tree& t) {
    const Dims d = dims(rows, cols);
    static_assert(sizeof(zl::Head) % 16 == 0, "nodes are read as uint4");
    char* z = (char*)zim_scratch_take(ctx, d.zeroed);
    t.leaf = (float4*)zim_scratch_take(ctx, d.leaf);
    if (!z || !t.leaf) return zim_fail(ctx, ZIM_ERR_OUT_OF_MEMORY, "leaf tree scratch");
    t.head = (zl::Head*)z;
    t.node = (unsigned*)(z + sizeof(zl::Head));
    t.lw = d.lw; t.lh = d.lh; t.nw = d.nw; t.nh = d.nh;
    return ZIM_OK;
}

zim_status zim_leaf_build(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows, int cols,
                          const zt::RayParams* rays, zl::Tree& t, cudaStream_t st) {
    ZIM_CUDA_TRY(ctx, cudaMemsetAsync(t.head, 0, dims(rows, cols).zeroed, st));
    leaf_kernel<<<(unsigned)t.nw * (unsigned)t.lh, LB, 0, st>>>(xyz, mask, rows, cols, rays ? 1 : 0, rays ? *rays : zt::RayParams{},
                                                 t);
    ctx->launches += 1;
    ZIM_LAUNCH_CHECK(ctx);
    return ZIM_OK;
}
