// psb_voxel.cuh — mesh voxelizer: the caller-side input stage of the packer
// (the reference's voxelize_stl, spectral_packing/bindings.cpp:285-302 and
// packing.cpp:309-588, VoxSurf).
//
// The reference rasterizes every triangle along the three axes in 16-bit
// fixed point: for each pixel centre inside the projected triangle (64-bit
// edge functions) the voxel at the barycentric depth has its axis bit
// flipped; a pixel exactly on an edge counts for one of the two triangles
// sharing it (the one whose edge runs from the lower to the higher vertex
// index).  With the inside fill compiled out (constants.h:9) a voxel is
// occupied when any axis bit is set.  Flips commute, so pixels can be taken in
// any order and split freely: eight lanes walk a small triangle's pixel box
// along one axis and a larger one is cut into chunks of 256 pixels, a warp
// each (k_voxel_raster, k_voxel_chunks).
//
// The reference first merges equal vertices and numbers them in lexicographic
// order of their positions; the numbers are only ever compared, so here the
// positions themselves are (lex_less), and nothing is sorted: the host sort
// of 49,152 vertices was most of the 6 ms that a 16,384-triangle mesh took.
#pragma once
#include <stdint.h>

#include "psb_pdl.cuh"

#define PSB_FP_POW 16
#define PSB_FP_SCALE (1 << PSB_FP_POW)

// packing.cpp:309-335
__device__ __forceinline__ bool vox_in_triangle(long long i, long long j, const int* p0, const int* p1,
                                                const int* p2, int* depth, int* aligned) {
    const long long d0x = i - p0[0], d0y = j - p0[1];
    const long long d1x = i - p1[0], d1y = j - p1[1];
    const long long d2x = i - p2[0], d2y = j - p2[1];
    const long long e10x = (long long)p1[0] - p0[0], e10y = (long long)p1[1] - p0[1];
    const long long e21x = (long long)p2[0] - p1[0], e21y = (long long)p2[1] - p1[1];
    const long long e02x = (long long)p0[0] - p2[0], e02y = (long long)p0[1] - p2[1];
    const long long c0 = d0x * e10y - d0y * e10x;
    const long long c1 = d1x * e21y - d1y * e21x;
    const long long c2 = d2x * e02y - d2y * e02x;
    const bool inside = (c0 <= 0 && c1 <= 0 && c2 <= 0) || (c0 >= 0 && c1 >= 0 && c2 >= 0);
    *aligned = (c0 == 0) ? 0 : ((c1 == 0) ? 1 : ((c2 == 0) ? 2 : -1));
    if (inside) {
        const long long area = c0 + c1 + c2;
        const long long b0 = (c1 << 10) / area;   // truncating division, as in C++
        const long long b1 = (c2 << 10) / area;
        const long long b2 = (1LL << 10) - b0 - b1;
        *depth = (int)((b0 * p0[2] + b1 * p1[2] + b2 * p2[2]) >> 10);
    }
    return inside;
}

// std::array<float, 3>'s operator<
__device__ __forceinline__ bool lex_less(const float* p, const float* q) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (p[a] < q[a]) return true;
        if (q[a] < p[a]) return false;
    }
    return false;
}

// float order as unsigned order
__device__ __forceinline__ unsigned int vox_key(float f) {
    const unsigned int b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// Bounding box of the vertices: key[0..2] smallest, key[3..5] largest
// (vox_key; preset to ~0 and 0).  grid: any, block 256
__global__ void k_voxel_bounds(const float* __restrict__ tris, long long nv, unsigned int* __restrict__ key) {
    pdl_enter();
    unsigned int lo[3] = {~0u, ~0u, ~0u}, hi[3] = {0u, 0u, 0u};
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < nv; v += (long long)gridDim.x * blockDim.x)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const unsigned int k = vox_key(tris[3 * v + a]);
            lo[a] = min(lo[a], k);
            hi[a] = max(hi[a], k);
        }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = __reduce_min_sync(0xffffffffu, lo[a]);
        hi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&key[a], lo[a]);
            atomicMax(&key[3 + a], hi[a]);
        }
    }
}

// the box transform (rows of the 4x4 matrix) and its upper clamp
struct VoxBox {
    float m[3][4];
    float top;
};

// One triangle seen along one axis: its vertices as (u, v, depth) in fixed
// point, their order and the pixel box.
struct VoxView {
    int tp[3][3];
    bool less[3];               // vertex k sorts before vertex (k + 1) % 3
    int x0, y0, nx;
    long long npix;             // 0: degenerate
};

// Fixed-point vertices (products and sums rounded one by one, as LibSL's
// Matrix4x4 evaluates them) and the view's swizzle (packing.cpp:337-360):
//   view 0 xyz along z; view 1 yzx along x; view 2 zxy along y
__device__ __forceinline__ VoxView vox_view(const float* __restrict__ tris, int t, int view, const VoxBox& box) {
    VoxView w;
    float p[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int a = 0; a < 3; ++a) p[k][a] = __ldg(&tris[9 * (size_t)t + 3 * k + a]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        int c[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < 3; ++j) acc = __fadd_rn(acc, __fmul_rn(box.m[a][j], p[k][j]));
            acc = __fadd_rn(acc, box.m[a][3]);
            c[a] = (int)fminf(fmaxf(roundf(acc), 0.f), box.top);
        }
        w.tp[k][0] = view == 0 ? c[0] : (view == 1 ? c[1] : c[2]);
        w.tp[k][1] = view == 0 ? c[1] : (view == 1 ? c[2] : c[0]);
        w.tp[k][2] = view == 0 ? c[2] : (view == 1 ? c[0] : c[1]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) w.less[k] = lex_less(p[k], p[(k + 1) % 3]);
    const int (&tp)[3][3] = w.tp;
    w.npix = 0;
    const long long e10x = tp[1][0] - tp[0][0], e10y = tp[1][1] - tp[0][1];
    const long long e21x = tp[2][0] - tp[1][0], e21y = tp[2][1] - tp[1][1];
    const long long e02x = tp[0][0] - tp[2][0], e02y = tp[0][1] - tp[2][1];
    if ((e10x == 0 && e10y == 0) || (e21x == 0 && e21y == 0) || (e02x == 0 && e02y == 0)) return w;
    // the reference forms this determinant from 32-bit int products (v2i),
    // which wrap at these fixed-point magnitudes: a nonzero multiple of 2^32
    // counts as degenerate there, so it is evaluated modulo 2^32 here too
    // (a unit cube at a resolution where 0.95 * res is an integer loses every face)
    if ((unsigned int)e02x * (unsigned int)e10y - (unsigned int)e02y * (unsigned int)e10x == 0u) return w;
    w.x0 = min(tp[0][0], min(tp[1][0], tp[2][0])) / PSB_FP_SCALE;
    const int x1 = max(tp[0][0], max(tp[1][0], tp[2][0])) / PSB_FP_SCALE;
    w.y0 = min(tp[0][1], min(tp[1][1], tp[2][1])) / PSB_FP_SCALE;
    const int y1 = max(tp[0][1], max(tp[1][1], tp[2][1])) / PSB_FP_SCALE;
    w.nx = x1 - w.x0 + 1;
    w.npix = (long long)w.nx * (y1 - w.y0 + 1);
    return w;
}

// pixel q of the view's box
__device__ __forceinline__ void vox_pixel(const VoxView& w, int view, long long q, int X, int Y, int Z,
                                          unsigned int* __restrict__ vox) {
    const int i = w.x0 + (int)(q % w.nx), j = w.y0 + (int)(q / w.nx);
    int depth = 0, aligned = -1;
    if (!vox_in_triangle(((long long)i << PSB_FP_POW) + (1 << (PSB_FP_POW - 1)),
                         ((long long)j << PSB_FP_POW) + (1 << (PSB_FP_POW - 1)), w.tp[0], w.tp[1], w.tp[2], &depth,
                         &aligned))
        return;
    if (aligned != -1 && !w.less[aligned]) return;
    const int d = depth >> PSB_FP_POW;
    // backward swizzle
    const int v0 = view == 0 ? i : (view == 1 ? d : j);
    const int v1 = view == 0 ? j : (view == 1 ? i : d);
    const int v2 = view == 0 ? d : (view == 1 ? j : i);
    if (v0 < 0 || v1 < 0 || v2 < 0 || v0 >= X || v1 >= Y || v2 >= Z) return;
    atomicXor(&vox[((size_t)v0 * Y + v1) * Z + v2], view == 0 ? 4u : (view == 1 ? 1u : 2u));
}

#define PSB_VCHUNK 256          // pixels per chunk of a large triangle
#define PSB_VCHUNKS (1 << 18)   // chunk list entries
// Eight lanes per (triangle, view); a pixel box above one chunk goes to the
// chunk list instead ({3 t + view, first chunk number}), or is walked here when
// the list is full.  grid: ceil(24 m / 256), block 256
__global__ void __launch_bounds__(256)
k_voxel_raster(const float* __restrict__ tris, int m, VoxBox box, int X, int Y, int Z, unsigned int* __restrict__ vox,
               int2* __restrict__ chunks, unsigned long long* __restrict__ nchunks) {
    pdl_enter();
    const long long g = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const int sub = threadIdx.x & 7;
    const bool in = g < 3LL * m;
    const int t = in ? (int)(g / 3) : 0, view = in ? (int)(g % 3) : 0;
    const VoxView w = vox_view(tris, t, view, box);
    const unsigned int group = 0xffu << (threadIdx.x & 24);
    long long npix = in ? w.npix : 0;
    if (npix > PSB_VCHUNK) {
        const int need = (int)((npix + PSB_VCHUNK - 1) / PSB_VCHUNK);
        unsigned long long first = 0;
        if (sub == 0) first = atomicAdd(nchunks, (unsigned long long)need);
        first = __shfl_sync(group, first, threadIdx.x & 24);
        const int at = (int)min(first, (unsigned long long)PSB_VCHUNKS);
        if (at <= PSB_VCHUNKS - need) {
            for (int k = sub; k < need; k += 8) chunks[at + k] = make_int2((int)g, k);
            npix = 0;
        } else if (sub == 0 && at < PSB_VCHUNKS) {
            // the entries between the list's last use and its end stay unused
            for (int k = at; k < PSB_VCHUNKS; ++k) chunks[k] = make_int2(-1, 0);
        }
    }
    for (long long q = sub; q < npix; q += 8) vox_pixel(w, view, q, X, Y, Z, vox);
}

// One warp per listed chunk.  grid: any, block 256
__global__ void __launch_bounds__(256)
k_voxel_chunks(const float* __restrict__ tris, VoxBox box, int X, int Y, int Z, unsigned int* __restrict__ vox,
               const int2* __restrict__ chunks, const unsigned long long* __restrict__ nchunks) {
    pdl_enter();
    const int n = (int)min(*nchunks, (unsigned long long)PSB_VCHUNKS);
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (int c = blockIdx.x * wpb + (threadIdx.x >> 5); c < n; c += gridDim.x * wpb) {
        const int2 h = chunks[c];
        if (h.x < 0) continue;
        const VoxView w = vox_view(tris, h.x / 3, h.x % 3, box);
        const long long q1 = min(w.npix, ((long long)h.y + 1) * PSB_VCHUNK);
        for (long long q = (long long)h.y * PSB_VCHUNK + lane; q < q1; q += 32) vox_pixel(w, h.x % 3, q, X, Y, Z, vox);
    }
}

// Bounding box of the occupied voxels: b[0..2] smallest, b[3..5] largest
// (preset to INT_MAX and -1).  A warp per z line.  grid: any, block 256
__global__ void k_voxel_box(const unsigned int* __restrict__ vox, int X, int Y, int Z, int* __restrict__ b) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const long long nl = (long long)X * Y, step = (long long)gridDim.x * (blockDim.x >> 5);
    int lo[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, hi[3] = {-1, -1, -1};
    for (long long l = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); l < nl; l += step) {
        const int i = (int)(l / Y), j = (int)(l % Y);
        for (int k = lane; k < Z; k += 32)
            if (vox[l * Z + k]) {
                lo[0] = min(lo[0], i); hi[0] = max(hi[0], i);
                lo[1] = min(lo[1], j); hi[1] = max(hi[1], j);
                lo[2] = min(lo[2], k); hi[2] = max(hi[2], k);
            }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = __reduce_min_sync(0xffffffffu, lo[a]);
        hi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
        if (lane == 0 && hi[a] >= 0) {
            atomicMin(&b[a], lo[a]);
            atomicMax(&b[3 + a], hi[a]);
        }
    }
}

// The tight 0/1 grid (make_voxel_grid_tight) of extent (t0, t1, t2) from
// (l0, l1, l2) on, a warp per z line.  grid: any, block 256
__global__ void k_voxel_tight(const unsigned int* __restrict__ vox, int Y, int Z, int l0, int l1, int l2, int t0, int t1,
                              int t2, int32_t* __restrict__ out) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const long long nl = (long long)t0 * t1, step = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long l = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); l < nl; l += step) {
        const unsigned int* src = vox + ((size_t)(l / t1 + l0) * Y + (l % t1 + l1)) * Z + l2;
        for (int k = lane; k < t2; k += 32) out[l * t2 + k] = src[k] ? 1 : 0;
    }
}
