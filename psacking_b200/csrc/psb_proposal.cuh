// psb_proposal.cuh — the learned orientation proposal: a small 3-D CNN that
// ranks an item's orientations before the exact search.
//
// Network (parameters in one flat FP32 master vector, BF16 copies of the
// weights for the forward and backward passes, FP32 accumulation):
//   item branch, per orientation, 32^3 occupancy grid:
//     conv3d 1->16, 16->32, 32->64, 64->64 (kernel 3, stride 2, padding 1,
//     ReLU) -> 64 x 2^3 = 512 -> linear 512->64, ReLU
//   tray branch, per item, 32x32 pooled height map: linear 1024->64, ReLU
//   head, per orientation: [item 64 | tray 64] -> linear 128->64, ReLU ->
//     linear 64->1 = logit
// Loss: masked softmax cross-entropy over an item's orientations against a
// soft target from the plain search (weight 2^-rank by exact score among the
// orientations that fit somewhere), mean over the items that have one.
// Training and inference use the same kernels; the packing loop runs the
// forward pass on the device and keeps only the top-k orientations (all of
// them when the top-k probability mass is below a margin).
// No counterpart in the reference: the learned-proposal form is an addition.
#pragma once
#include <stdint.h>

#include "psb_conv.cuh"

#define PSB_PG 32          // item grid side
#define PSB_PG3 (PSB_PG * PSB_PG * PSB_PG)
#define PSB_PH 32          // pooled height-map side
#define PSB_PNO 24         // orientations per item in the network's output

// BF16 storage as uint16 (round to nearest even; inputs are finite)
__host__ __device__ __forceinline__ uint16_t bf16_bits(float f) {
#ifdef __CUDA_ARCH__
    uint32_t u = __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, 4);
#endif
    u += 0x7fffu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}
__device__ __forceinline__ float bf16_val(uint16_t h) { return bf16_up(h); }

// ---------------------------------------------------------------------------
// inputs
// ---------------------------------------------------------------------------
// base grids of items given as dense arrays (the synchronous item-grid call;
// the packing loop uses k_base_grid_runs): cell (i, j, k) of an item holds the
// occupied fraction of its s^3 block, s = ceil(max extent / 32), summed voxel
// by voxel as the runs form does.  One thread per cell, no atomics.
// grid: (PSB_PG3 / 256, items), block 256
struct GridItem {
    long long off;              // the item's first value in `vals`
    int d[3], s;
};
__global__ void k_base_grid_dense(const int32_t* __restrict__ vals, const GridItem* __restrict__ items,
                                  float* __restrict__ out) {
    pdl_enter();
    const GridItem it = items[blockIdx.y];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int i0 = c / (PSB_PG * PSB_PG) * it.s, j0 = c / PSB_PG % PSB_PG * it.s, k0 = c % PSB_PG * it.s;
    const float w = 1.0f / (float)(it.s * it.s * it.s);
    float v = 0.f;
    const int32_t* a = vals + it.off;
    for (int i = i0; i < min(i0 + it.s, it.d[0]); ++i)
        for (int j = j0; j < min(j0 + it.s, it.d[1]); ++j)
            for (int k = k0; k < min(k0 + it.s, it.d[2]); ++k)
                if (__ldg(&a[((size_t)i * it.d[1] + j) * it.d[2] + k]) > 0) v += w;
    out[(size_t)blockIdx.y * PSB_PG3 + c] = v;
}

// the base grid of one item from its z-runs ({x, y, z0 | z1 << 16, value},
// one per run of equal nonzero values along z): cell floor(v / s) gains 1/s^3
// per voxel.  grid: (ceil(nruns/256)), block 256; out zeroed
__global__ void k_base_grid_runs(const int4* __restrict__ runs, int nruns, int s, float* __restrict__ out) {
    pdl_enter();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nruns) return;
    const int4 q = runs[r];
    if (q.w <= 0) return;
    const float w = 1.0f / (float)(s * s * s);
    const int i = q.x / s, j = q.y / s, z1 = q.z >> 16;
    for (int z = q.z & 0xffff; z <= z1; ++z) atomicAdd(&out[(i * PSB_PG + j) * PSB_PG + z / s], w);
}

// oriented grids: out[b*no + o] = the base grid of item b turned by map o
// (src_axis[3], flip[3]) within its scaled extent G (cells per axis).  Bound by
// the store of no times the base grids; four z cells per thread, one 16-byte
// store (one cell per thread: 206 us at 64 items x 24, the index arithmetic and
// a warp instruction per 128 bytes).
// grid: (PSB_PG3 / 1024, no, B), block 256
__global__ void k_orient_grids(const float* __restrict__ base, const int* __restrict__ G, const int* __restrict__ maps,
                               int no, float* __restrict__ out) {
    pdl_enter();
    const int b = blockIdx.z, o = blockIdx.y;
    const int c = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (c >= PSB_PG3) return;
    const int* m = maps + 6 * o;
    const int ijk[3] = {c / (PSB_PG * PSB_PG), (c / PSB_PG) % PSB_PG, c % PSB_PG};
    const int str[3] = {PSB_PG * PSB_PG, PSB_PG, 1};
    int at = 0, dz = 0, n = 0;   // source of the first cell, its step, cells inside
    bool in = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int sa = m[a], st = str[sa], ga = G[3 * b + sa];
        in = in && ijk[a] < ga;
        at += (m[3 + a] ? ga - 1 - ijk[a] : ijk[a]) * st;
        if (a == 2) {
            dz = m[3 + a] ? -st : st;
            n = min(4, ga - ijk[a]);
        }
    }
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (in) {
        const float* p = base + (size_t)b * PSB_PG3 + at;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < n) v[k] = p[k * dz];
    }
    float* q = out + ((size_t)b * no + o) * PSB_PG3 + c;
    if (((uintptr_t)out & 15) == 0) {   // else the caller's buffer starts between 16-byte boundaries
        *(float4*)q = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = v[k];
    }
}

// pooled height map: per column 1 + highest occupied z (0 when empty), over
// nz, averaged over ceil(nx/32) x ceil(ny/32) blocks.  One CTA per pooled
// cell, one warp per column at a time: lanes read 32 consecutive z from the
// top down and a ballot finds the highest occupied one.
// grid: 1024, block 256
__global__ void k_height_map(const int32_t* __restrict__ tray, int nx, int ny, int nz, float* __restrict__ out) {
    pdl_enter();
    const int cell = blockIdx.x;  // 0..1023
    const int ci = cell / PSB_PH, cj = cell % PSB_PH;
    const int bx = (nx + PSB_PH - 1) / PSB_PH, by = (ny + PSB_PH - 1) / PSB_PH;
    const int x0 = ci * bx, y0 = cj * by;
    const int x1 = min(nx, x0 + bx), y1 = min(ny, y0 + by);
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nwp = blockDim.x >> 5;
    __shared__ float red[8];
    __shared__ int cnt[8];
    float acc = 0.f;
    int n = 0;
    const int w = max(0, y1 - y0);
    const int ncol = max(0, x1 - x0) * w;
    for (int c = wp; c < ncol; c += nwp) {
        const int x = x0 + c / w, y = y0 + c % w;
        const int32_t* col = tray + ((size_t)x * ny + y) * nz;
        int top = 0;
        for (int zb = ((nz - 1) / 32) * 32; zb >= 0; zb -= 32) {
            const int z = zb + lane;
            const unsigned int bal = __ballot_sync(0xffffffffu, z < nz && col[z] > 0);
            if (bal) {
                top = zb + 32 - __clz(bal);
                break;
            }
        }
        acc += (float)top / (float)nz;
        ++n;
    }
    if (lane == 0) {
        red[wp] = acc;
        cnt[wp] = n;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
        int k = 0;
        for (int i = 0; i < nwp; ++i) { s += red[i]; k += cnt[i]; }
        out[cell] = k ? s / (float)k : 0.f;
    }
}

// head input: [f1[s] | t[s / no]] (64 + 64).  grid: ceil(S*128/256)
__global__ void k_concat(const float* __restrict__ f1, const float* __restrict__ t, int S, int no, float* __restrict__ hin) {
    pdl_enter();
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)S * 128) return;
    const int s = (int)(idx / 128), c = (int)(idx % 128);
    hin[idx] = c < 64 ? f1[(size_t)s * 64 + c] : t[(size_t)(s / no) * 64 + (c - 64)];
}

// split the head-input gradient: df1 = dhin[:, :64] * (f1 > 0);
// dt[b] = sum over its orientations of dhin[:, 64:] * (t > 0).  grid: ceil(S*64/256) and ceil(B*64/256)
__global__ void k_split_item(const float* __restrict__ dhin, const float* __restrict__ f1, int S,
                             float* __restrict__ df1) {
    pdl_enter();
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)S * 64) return;
    const int s = (int)(idx / 64), c = (int)(idx % 64);
    df1[idx] = f1[idx] > 0.f ? dhin[(size_t)s * 128 + c] : 0.f;
}
__global__ void k_split_tray(const float* __restrict__ dhin, const float* __restrict__ t, int B, int no,
                             float* __restrict__ dt) {
    pdl_enter();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= B * 64) return;
    const int b = idx / 64, c = idx % 64;
    float acc = 0.f;
    for (int o = 0; o < no; ++o) acc += dhin[((size_t)b * no + o) * 128 + 64 + c];
    dt[idx] = t[idx] > 0.f ? acc : 0.f;
}

// masked softmax cross-entropy over each item's no logits, mean over the
// items that have a target and an unmasked orientation; loss accumulated in
// *loss (zeroed first), gradient written to dlogit.  One warp per item.
__global__ void k_softmax_ce(const float* __restrict__ logit, const float* __restrict__ target,
                             const float* __restrict__ mask, int B, int no, float* __restrict__ dlogit,
                             float* __restrict__ loss) {
    pdl_enter();
    const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    // items counted in the mean (the same for every warp)
    int nb = 0;
    for (int i = lane; i < B; i += 32) {
        float ts = 0.f, ms = 0.f;
        for (int o = 0; o < no; ++o) { ts += target[(size_t)i * no + o]; ms += mask[(size_t)i * no + o]; }
        nb += (ts > 0.f && ms > 0.f) ? 1 : 0;
    }
    nb = __reduce_add_sync(0xffffffffu, nb);
    if (b >= B) return;
    const float inv = 1.f / (float)max(1, nb);
    const bool m = lane < no && mask[(size_t)b * no + lane] > 0.f;
    const float z = m ? logit[(size_t)b * no + lane] : -INFINITY;
    float zmax = z;
    for (int off = 16; off > 0; off >>= 1) zmax = fmaxf(zmax, __shfl_xor_sync(0xffffffffu, zmax, off));
    const float e = m ? expf(z - zmax) : 0.f;
    float s = e;
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    const float q = (lane < no) ? target[(size_t)b * no + lane] : 0.f;
    float qs = q;
    for (int off = 16; off > 0; off >>= 1) qs += __shfl_xor_sync(0xffffffffu, qs, off);
    int anym = __any_sync(0xffffffffu, m);
    const bool has = qs > 0.f && anym;
    float lterm = 0.f, g = 0.f;
    if (has && m) {
        const float p = e / s;
        lterm = -q * (z - zmax - logf(s));
        g = (p * qs - q) * inv;
    }
    if (lane < no) dlogit[(size_t)b * no + lane] = g;
    for (int off = 16; off > 0; off >>= 1) lterm += __shfl_xor_sync(0xffffffffu, lterm, off);
    if (lane == 0 && has) atomicAdd(loss, lterm * inv);
}

// Adam on the FP32 master vector; weights (flag 1) get their BF16 copy
// refreshed.  grid: ceil(n/256)
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       uint16_t* __restrict__ p16, const unsigned char* __restrict__ is_weight, long long n, float lr,
                       float b1, float b2, float eps, float c1, float c2) {
    pdl_enter();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pi;
    if (is_weight[i]) p16[i] = bf16_bits(pi);
}

// ---------------------------------------------------------------------------
// per-item head in the packing loop (the item branch is precomputed for the
// whole run: it does not depend on the tray state)
// ---------------------------------------------------------------------------
// Tray features of one item: t[n] = relu(hmap . W2[n] + b2[n]), one CTA per
// output.  grid: 64, block 256
__global__ void k_prop_tray_feat(const float* __restrict__ hmap, const uint16_t* __restrict__ w2,
                                 const float* __restrict__ b2, float* __restrict__ t) {
    pdl_enter();
    const int n = blockIdx.x;
    float acc = 0.f;
    for (int k = threadIdx.x; k < PSB_PH * PSB_PH; k += blockDim.x)
        acc = fmaf(hmap[k], bf16_val(w2[(size_t)n * PSB_PH * PSB_PH + k]), acc);
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    __shared__ float red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float v = b2[n];
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) v += red[i];
        t[n] = fmaxf(v, 0.f);
    }
}

// Head of one item: per orientation o (one CTA), h1 = relu([f1_o | t] H1^T +
// bh1) (64 threads) and logit_o = h1 . H2 + bh2.  grid: no, block 64
__global__ void k_prop_item_head(const float* __restrict__ f1, const float* __restrict__ t,
                                 const uint16_t* __restrict__ wh1, const float* __restrict__ bh1,
                                 const uint16_t* __restrict__ wh2, const float* __restrict__ bh2,
                                 float* __restrict__ logit) {
    pdl_enter();
    const int o = blockIdx.x, n = threadIdx.x;
    __shared__ float in[128];
    __shared__ float red[2];
    in[n] = f1[(size_t)o * 64 + n];
    in[64 + n] = t[n];
    __syncthreads();
    const uint16_t* wr = wh1 + (size_t)n * 128;
    float acc = bh1[n];
    for (int k = 0; k < 128; ++k) acc = fmaf(in[k], bf16_val(wr[k]), acc);
    float v = fmaxf(acc, 0.f) * bf16_val(wh2[n]);
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((n & 31) == 0) red[n >> 5] = v;
    __syncthreads();
    if (n == 0) logit[o] = red[0] + red[1] + bh2[0];
}

// ---------------------------------------------------------------------------
// gating in the packing loop
// ---------------------------------------------------------------------------
// Keep the top-k orientations of one item by logit (ties: lower index), all
// of them when their softmax mass over the fitting orientations is below
// `margin`; the others are marked skipped for the search.  Orientations the
// tray cannot hold are skipped already.  One warp.
template <class OD>
__global__ void k_gate(const float* __restrict__ logit, OD* __restrict__ od, int n, int topk, float margin,
                       int* __restrict__ stats) {
    pdl_enter();
    const int lane = threadIdx.x;
    if (lane >= 32) return;
    const bool fit = lane < n && !od[lane].skip;
    const float z = fit ? logit[lane] : -INFINITY;
    float zmax = z;
    for (int off = 16; off > 0; off >>= 1) zmax = fmaxf(zmax, __shfl_xor_sync(0xffffffffu, zmax, off));
    const float e = fit ? expf(z - zmax) : 0.f;
    float s = e;
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    // rank of this orientation: how many fitting orientations beat it
    int rank = 0;
    for (int j = 0; j < 32; ++j) {
        const float zj = __shfl_sync(0xffffffffu, z, j);
        const bool fj = __shfl_sync(0xffffffffu, (int)fit, j) != 0;
        if (fj && (zj > z || (zj == z && j < lane))) ++rank;
    }
    const bool keep = fit && rank < topk;
    float mass = keep ? e / s : 0.f;
    for (int off = 16; off > 0; off >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, off);
    const bool fallback = mass < margin;
    if (fit && !keep && !fallback) od[lane].skip = 1;
    if (lane == 0 && stats) {
        atomicAdd(&stats[0], 1);
        if (fallback) atomicAdd(&stats[1], 1);
    }
}
