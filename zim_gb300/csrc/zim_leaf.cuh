// zim_leaf.cuh -- a two-level tree of bounding boxes over the valid points of
// an organised cloud: leaves of 8 x 8 pixels, nodes of 8 x 8 leaves.  Neighbours
// in space are mostly neighbours in the image, so the image itself is the
// spatial index: one pass over the cloud builds it, and no point is sorted or
// copied.  The searches (grid.cu) read the cloud through it.
//
// Box tests are exact without margins: a box holds the points' own float
// coordinates, float subtraction and fmaf round monotonically, so a box's
// rounded distance never exceeds the rounded distance of a point inside it
// (and its far corner's is never below one).
#pragma once

#include "zim_tiles.cuh"

namespace zl {

constexpr int LEAF = 8;             // leaf side in pixels
constexpr int FAN = 8;              // node side in leaves
constexpr int NODE = LEAF * FAN;    // node side in pixels

// Counters of one filter run, zeroed before the build.
struct Head {
    unsigned n_valid;       // valid points
    unsigned ray_dev_bits;  // largest distance of a point from its pixel ray (float bits)
    unsigned n_deferred;    // queries a window pass left to the tree
    unsigned next;          // work counter of the tree search
    unsigned done;          // finished blocks of the last reduction
    unsigned pad[3];
};

// Boxes are two float4 each: (lo, finite points as int bits), (hi, largest ray
// distance); an empty one has lo = +inf, hi = -inf.
struct Tree {
    Head* head;
    float4 *node, *leaf;
    int lw, lh, nw, nh;
};

// Order-preserving unsigned key of a float; 0 is below every float's key.
__device__ __forceinline__ unsigned fkey(float f) {
    const unsigned b = __float_as_uint(f);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float keyf(unsigned k) { return __uint_as_float(k & 0x80000000u ? k & 0x7fffffffu : ~k); }

struct Box {
    float lo[3], hi[3];
    unsigned n;
};

__device__ __forceinline__ Box load_box(const float4* boxes, int i) {
    const float4 a = __ldg(boxes + 2 * (size_t)i), b = __ldg(boxes + 2 * (size_t)i + 1);
    return Box{{a.x, a.y, a.z}, {b.x, b.y, b.z}, __float_as_uint(a.w)};
}

// Points with a NaN or infinite coordinate are nobody's neighbour: outside every box,
// window and grid.
__device__ __forceinline__ bool finite_point(float x, float y, float z) {
    return fmaf(x, 0.f, fmaf(y, 0.f, z * 0.f)) == 0.f;
}

__device__ __forceinline__ float sq3(float dx, float dy, float dz) { return fmaf(dz, dz, fmaf(dy, dy, dx * dx)); }

// Squared distance between the box and the box [lo, hi] (a point: lo = hi).
__device__ __forceinline__ float gap_d2(const Box& b, const float (&lo)[3], const float (&hi)[3]) {
    float e[3];
#pragma unroll
    for (int a = 0; a < 3; a++) e[a] = fmaxf(fmaxf(b.lo[a] - hi[a], lo[a] - b.hi[a]), 0.f);
    return sq3(e[0], e[1], e[2]);
}
// Squared distance from q to the box's farthest corner.
__device__ __forceinline__ float far_d2(const Box& b, const float (&q)[3]) {
    float e[3];
#pragma unroll
    for (int a = 0; a < 3; a++) e[a] = fmaxf(fabsf(b.lo[a] - q[a]), fabsf(b.hi[a] - q[a]));
    return sq3(e[0], e[1], e[2]);
}

// Leaf index of child c (0..63) of node n, -1 outside the image.
__device__ __forceinline__ int child_leaf(const Tree& t, int n, int c) {
    const int lx = (n % t.nw) * FAN + (c & (FAN - 1)), ly = (n / t.nw) * FAN + (c / FAN);
    return lx < t.lw && ly < t.lh ? ly * t.lw + lx : -1;
}

}  // namespace zl

// Scratch of a rows x cols cloud's tree; its carving; its build (one memset and
// one kernel).  With pixel rays the leaves and the head also hold the largest
// distance of a point from its ray.
size_t zim_leaf_bytes(int rows, int cols);
zim_status zim_leaf_carve(zim_ctx* ctx, int rows, int cols, zl::Tree& t);
zim_status zim_leaf_build(zim_ctx* ctx, const float* xyz, const uint8_t* mask, int rows, int cols,
                          const zt::RayParams* rays, zl::Tree& t, cudaStream_t st);
