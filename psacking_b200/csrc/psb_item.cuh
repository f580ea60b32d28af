// psb_item.cuh — the analysis of items handed to the synchronous searches as
// dense arrays: z-runs, sums, bounds, filter samples and the orientation
// descriptor itself, on the device (the packing loop's items are analysed on
// the host cores while the loop runs, build_runs and pick_samples).  On the
// host this was a pass per orientation building a 16-byte voxel list, most of
// the 8 ms a 24-orientation batch spent outside its kernels.
#pragma once
#include "psb_filter.cuh"

// One array: its values, the room for its runs and its dims.
struct ItemArr {
    long long off;              // first value in `vals`
    long long roff, room;       // first entry in `runs`, entries there
    int d[3];
    int skip;                   // larger than the tray
};

// What the runs pass collects per array.
struct ItemSums {
    double sumsq;
    long long sum;
    int nvox, nruns, neg;
    int lo[3], hi[3];           // bounds of the values > 0
};

// What the host reads back after a synchronous search by score bounds.
struct BoundReply {
    BoundState st;
    DecisionDev dec;
    int neg;                    // first array with a negative value, INT_MAX: none
};

__global__ void k_item_reset(ItemSums* s, int n, int* neg) {
    pdl_enter();
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o == 0) *neg = INT_MAX;
    if (o >= n) return;
    ItemSums z;
    z.sumsq = 0.0;
    z.sum = 0;
    z.nvox = z.nruns = z.neg = 0;
    for (int a = 0; a < 3; ++a) { z.lo[a] = INT_MAX; z.hi[a] = -1; }
    s[o] = z;
}

// The runs of equal nonzero values along z of every column, one warp per
// column: a cell starts a run when its value differs from the one below, ends
// one when it differs from the one above, and the k-th start of a column
// belongs to its k-th end, so starts and ends write their halves of the entry
// on their own.  A column's entries are reserved with one atomic (their order
// differs from call to call; every use sums over them).
// grid: (any, n), block 256
__global__ void __launch_bounds__(256)
k_item_runs(const int32_t* __restrict__ vals, const ItemArr* __restrict__ arrs, int4* __restrict__ runs,
            ItemSums* __restrict__ sums) {
    pdl_enter();
    const ItemArr it = arrs[blockIdx.y];
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    const long long ncol = (long long)it.d[0] * it.d[1];
    const int ez = it.d[2];
    const unsigned int below = (1u << lane) - 1u;
    ItemSums* S = sums + blockIdx.y;
    int4* R = runs + it.roff;
    double sumsq = 0.0;
    long long sum = 0;
    int nvox = 0, neg = 0;
    int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {-1, -1, -1};
    for (long long c = blockIdx.x * wpb + (threadIdx.x >> 5); c < ncol; c += gridDim.x * wpb) {
        const int32_t* col = vals + it.off + (size_t)c * ez;
        const int i = c >> 31 ? (int)(c / it.d[1]) : (int)c / it.d[1], j = (int)(c - (long long)i * it.d[1]);
        int cnt = 0;
        for (int z0 = 0; z0 < ez; z0 += 32) {
            const int z = z0 + lane;
            const int v = z < ez ? __ldg(&col[z]) : 0;
            const int p = z > 0 && z < ez ? __ldg(&col[z - 1]) : 0;
            cnt += __popc(__ballot_sync(0xffffffffu, v != 0 && v != p));
            if (v == 0) continue;
            ++nvox;
            sum += v;
            sumsq += (double)v * (double)v;
            neg |= v < 0;
            if (v > 0) {
                lo[0] = min(lo[0], i); hi[0] = max(hi[0], i);
                lo[1] = min(lo[1], j); hi[1] = max(hi[1], j);
                lo[2] = min(lo[2], z); hi[2] = max(hi[2], z);
            }
        }
        if (cnt == 0) continue;
        int base = 0;
        if (lane == 0) base = atomicAdd(&S->nruns, cnt);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base + cnt > it.room) continue;   // cannot be, unless the array changed while it was counted
        int s = base, e = base;
        for (int z0 = 0; z0 < ez; z0 += 32) {
            const int z = z0 + lane;
            const int v = z < ez ? __ldg(&col[z]) : 0;
            const int p = z > 0 && z < ez ? __ldg(&col[z - 1]) : 0;
            const int n = z + 1 < ez ? __ldg(&col[z + 1]) : 0;
            const unsigned int bs = __ballot_sync(0xffffffffu, v != 0 && v != p);
            const unsigned int be = __ballot_sync(0xffffffffu, v != 0 && v != n);
            if (v != 0 && v != p) {
                int4* r = R + s + __popc(bs & below);
                r->x = i;
                r->y = j;
                r->w = v;
                ((unsigned short*)&r->z)[0] = (unsigned short)z;
            }
            if (v != 0 && v != n) ((unsigned short*)&R[e + __popc(be & below)].z)[1] = (unsigned short)z;
            s += __popc(bs);
            e += __popc(be);
        }
    }
    nvox = __reduce_add_sync(0xffffffffu, nvox);
    if (nvox == 0) return;
    for (int d = 16; d > 0; d >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, d);
        sumsq += __shfl_xor_sync(0xffffffffu, sumsq, d);
    }
    neg = __any_sync(0xffffffffu, neg);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = __reduce_min_sync(0xffffffffu, lo[a]);
        hi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
    }
    if (lane != 0) return;
    atomicAdd(&S->nvox, nvox);
    atomicAdd((unsigned long long*)&S->sum, (unsigned long long)sum);
    atomicAdd(&S->sumsq, sumsq);
    if (neg) atomicOr(&S->neg, 1);
    for (int a = 0; a < 3; ++a) {
        atomicMin(&S->lo[a], lo[a]);
        atomicMax(&S->hi[a], hi[a]);
    }
}

// cells of a 5 x 5 x 5 split in farthest-point order from a corner (filled by
// the host), so the filter's first samples span the item
#define PSB_ICELLS 125
__constant__ unsigned char c_cell_order[PSB_ICELLS];

// Samples and descriptor of every array.  Sample: in each cell of a 5 x 5 x 5
// split of the box the voxel farthest from the centre (within a run and a cell
// that is one of the part's ends), in the order above; any subset of the voxels
// is exact for the filter.  grid: n, block 256
__global__ void __launch_bounds__(256)
k_item_describe(const int32_t* __restrict__ vals, const ItemArr* __restrict__ arrs, const int4* __restrict__ runs,
                const ItemSums* __restrict__ sums, int nx, int ny, int nz, int4* __restrict__ samp,
                OrientDesc* __restrict__ out, int* neg) {
    pdl_enter();
    __shared__ unsigned long long best[PSB_ICELLS];
    const int o = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const ItemArr it = arrs[o];
    ItemSums S = sums[o];
    S.nruns = (int)min((long long)S.nruns, it.room);
    const int4* R = runs + it.roff;
    for (int i = tid; i < PSB_ICELLS; i += 256) best[i] = 0ULL;
    __syncthreads();
    for (int r = tid; r < (it.skip ? 0 : S.nruns); r += 256) {
        const int4 q = R[r];
        if (q.w <= 0) continue;
        const int z1 = q.z >> 16;
        const int cij = (q.x * 5 / it.d[0] * 5 + q.y * 5 / it.d[1]) * 5;
        const int ax = 2 * q.x - it.d[0] + 1, ay = 2 * q.y - it.d[1] + 1;
        for (int k = q.z & 0xffff; k <= z1;) {
            const int c = k * 5 / it.d[2];
            const int e = min(z1, ((c + 1) * it.d[2] + 4) / 5 - 1);   // last z of the cell
            for (int u = 0; u < 2; ++u) {
                const int z = u ? e : k, az = 2 * z - it.d[2] + 1;
                const unsigned long long key = (unsigned long long)(unsigned int)(ax * ax + ay * ay + az * az) << 32 |
                                               (unsigned int)(q.x | q.y << 10 | z << 20) | 1ULL << 31;
                atomicMax(&best[cij + c], key);
            }
            k = e + 1;
        }
    }
    __syncthreads();
    if (tid >= 32) return;
    int4* P = samp + (size_t)o * PSB_FSAMP;
    int ns = 0;
    for (int i0 = 0; i0 < PSB_ICELLS; i0 += 32) {
        const unsigned long long k = i0 + lane < PSB_ICELLS ? best[c_cell_order[i0 + lane]] : 0ULL;
        const unsigned int b = __ballot_sync(0xffffffffu, k != 0ULL);
        if (k) {
            const unsigned int u = (unsigned int)k & 0x7fffffffu;
            P[ns + __popc(b & ((1u << lane) - 1u))] = make_int4(u & 1023, u >> 10 & 1023, u >> 20, 1);
        }
        ns += __popc(b);
    }
    if (lane != 0) return;
    const int n[3] = {nx, ny, nz};
    OrientDesc d;
    // an array with a negative value is an error that the host reads only after
    // the search: it is not searched, since its numbers of translations come
    // from its positive voxels and do not keep the negative ones inside
    d.skip = it.skip || S.neg;
    if (S.neg) atomicMin(neg, o);
    const bool empty = S.hi[0] < 0;
    for (int a = 0; a < 3; ++a) {
        d.src_axis[a] = a;
        d.flip[a] = 0;
        d.b[a] = d.e[a] = it.d[a];
        d.hi[a] = empty ? -1 : S.hi[a];
        d.valid[a] = empty ? n[a] : max(0, n[a] - d.hi[a]);
    }
    d.exact = 0;
    d.sumI = d.sabs = S.sum;
    d.delta = d.base = 0.0;     // k_prep
    d.item = vals + it.off;
    d.nvox = S.nvox;
    d.perm = -1;
    d.sumsq = S.sumsq;
    d.samp = P;
    d.nsamp = ns;
    d.direct = 0;
    d.runs = R;
    d.nruns = S.nruns;
    out[o] = d;
}

// Placement of an item in a resident tray: the first tray cell (row-major)
// where it meets an occupied one (WRITE false), then, when there is none, the
// cells written (packing.cpp:773-788).  Over the dense item, since a run's ends
// are 16 bits wide and the item may be longer than the tray (parts outside are
// left out): tray box of n cells from lo on, which lies at off in the item.
// grid: any, block 256
struct PlaceBox {
    int lo[3], n[3], off[3];
};
template <bool WRITE>
__global__ void k_place_dense(const int32_t* __restrict__ item, int ey, int ez, int32_t* __restrict__ tray, int ny, int nz,
                              PlaceBox b, int32_t id, unsigned long long* first) {
    pdl_enter();
    const size_t m = (size_t)b.n[0] * b.n[1] * b.n[2];
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < m; t += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(t % b.n[2]), j = (int)(t / b.n[2] % b.n[1]), i = (int)(t / ((size_t)b.n[2] * b.n[1]));
        if (__ldg(&item[((size_t)(i + b.off[0]) * ey + (j + b.off[1])) * ez + k + b.off[2]]) <= 0) continue;
        const size_t c = ((size_t)(i + b.lo[0]) * ny + (j + b.lo[1])) * nz + k + b.lo[2];
        if (WRITE) {
            if (tray[c] == 0) tray[c] = id;
        } else if (tray[c] > 0) {
            atomicMin(first, (unsigned long long)c);
        }
    }
}

// place_in_tray on a box of the tray: item value > 0 on an occupied cell gives
// the first overlap, on an empty one writes the id.  box (bx, by, bz) at
// (ox, oy, oz) of the item (ex, ey, ez); out receives the box.
// grid: any, block 256
__global__ void k_place_box(const int32_t* __restrict__ box, int bx, int by, int bz, const int32_t* __restrict__ item, int ey,
                            int ez, int ox, int oy, int oz, int32_t id, int32_t* __restrict__ out,
                            unsigned long long* first) {
    pdl_enter();
    const size_t n = (size_t)bx * by * bz;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(t % bz), j = (int)(t / bz % by), i = (int)(t / ((size_t)bz * by));
        int v = box[t];
        if (item[((size_t)(i + ox) * ey + (j + oy)) * ez + k + oz] > 0) {
            if (v > 0) atomicMin(first, (unsigned long long)t);
            else if (v == 0) v = id;
        }
        out[t] = v;
    }
}
