// psb_bound.cuh — the packing search by exact score bounds, without transforms.
//
// An item's winner is the free translation with the smallest score
//   D(t) + penalty(z),   D(t) = sum over item voxels v of w(v) phi(t + v),
// phi the L1 distance to the tray's sources (the cells equal to 1).  Two
// lower bounds of D cost a few operations per translation, because phi is at
// least the L1 distance to any box or half space that holds every source:
//   * separable: phi(p) >= dx(px) + dy(py) + dz(pz), the distance to the
//     sources' bounding box, so D(t) >= X(x) + Y(y) + Z(z), each a sum over
//     one marginal of the item;
//   * octants: phi(p) >= s.p - h(s) for each sign vector s, h(s) the largest
//     s.q over the sources q, so D(t) >= W s.t + (s.M - W h(s)) with W the
//     item's total weight and M its first moment (equality where the whole
//     item lies beyond the sources in that octant).
// Both are exact integers, and a score grows with D at fixed z, so a
// translation whose bounded score exceeds a score already achieved cannot
// win.  Measured on packing runs (128^3 and 240x123x100 trays, 24
// orientations, 15-40 million translations per item), between 4 and a few
// thousand free translations of all orientations together stay below the
// winner's score; the transforms this replaces evaluated all of them.
//
// Per item:
//   1. k_bound_seed, on a lattice of every fourth column in x and y: the
//      bit-parallel sample filter (psb_filter.cuh) leaves the translations that
//      may be free, each warp checks and scores its lowest-bound survivor
//      exactly, and the item's best score so far comes down;
//      k_bound_find, on every column: the z range is cut where the
//      bounds exceed the best score, the filter runs on what is left, and the
//      survivors are listed;
//   2. k_bound_score: the listed translations whose bound still does not
//      exceed the best score are checked and scored exactly (integer sums), and
//      the last CTA picks the winner by the reference's tie rules.
// In the interlocking mode k_bound_ray then looks for a straight free run
// from the winner to a seed face, which proves it reachable (the reachable
// translations are a subset of the free ones, so the best free one is then
// the best reachable one).  Where there is none, k_bound_find (ALL) lists every
// survivor, k_bound_flood checks them and floods the free ones from the seed
// faces in one CTA's shared memory (a crowded tray has few), and a second
// k_bound_score takes the best reachable one.  k_bound_place writes the item.
// An item this cannot decide (no source, weights or distances too large for
// exact scores, more survivors than the list or free ones than the flood holds)
// raises BoundState::halt: the launches already queued for later items return at
// once, and the host runs that item through the transforms and the union-find
// flood fill.
#pragma once
#include "psb_filter.cuh"

#define PSB_BSTEP 4             // seed lattice in x
#define PSB_BCAP (1 << 16)      // listed translations per item
#define PSB_BFREE 8192          // free translations the shared-memory flood takes
#define PSB_BBATCH 16           // sample buckets are padded to whole batches of this many
#define PSB_BSAMP (PSB_FSAMP + 8 * (PSB_BBATCH - 1))
#define PSB_BHDR 16             // doubles before a table's X, Y, Z parts

// The distance sources (cells equal to 1): their bounding box and, per sign
// vector s (bit a of the index set: axis a negative), the largest s.q.
struct BoundGeom {
    int lo[3], hi[3];
    int h[8];
    int any;                    // a source exists
    int over;                   // largest excess of the bounds over phi (0 for a distance field)
    int pmax;                   // no value of phi is larger, or smaller than -pmax - 1
};

struct __align__(16) BoundState {
    unsigned long long best;    // ord_key of the best score so far of the current item
    int count;                  // listed translations
    int halt;
    int need_ray, need_flood;
    int nwin;                   // translations that were the best when scored
    unsigned int blocked;       // k_bound_ray: directions with a blocked cell
    double win_s;
    int win_o, win_t;
    unsigned int done, rdone;   // CTAs finished (k_bound_score / k_bound_flood, k_bound_ray)
    int halt_item;
    int pad;
};
// the part a kernel reads on entry, in two loads (each field on its own would
// be a dependent round trip to L2 before the work starts)
struct BoundEntry {
    double best;
    int count, halt, need_ray, need_flood, nwin;
};
__device__ __forceinline__ BoundEntry bound_entry(const BoundState* st) {
    const int4 a = __ldcg((const int4*)st), b = __ldcg((const int4*)st + 1);
    BoundEntry e;
    const unsigned long long k = (unsigned long long)(unsigned int)a.x | (unsigned long long)(unsigned int)a.y << 32;
    e.best = k == 0xffffffffffffffffULL ? INFINITY : ord_val(k);
    e.count = a.z;
    e.halt = a.w;
    e.need_ray = b.x;
    e.need_flood = b.y;
    e.nwin = b.z;
    return e;
}

struct BoundHit {
    int t, o;
    double s;                   // the bounded score, then the exact one
};

// pmax: 0 where k_bound_over follows
__global__ void k_bound_geom_reset(BoundGeom* g, int pmax) {
    pdl_enter();
    if (threadIdx.x != 0) return;
    for (int a = 0; a < 3; ++a) { g->lo[a] = INT_MAX; g->hi[a] = -1; }
    for (int k = 0; k < 8; ++k) g->h[k] = INT_MIN;
    g->any = 0;
    g->over = 0;
    g->pmax = pmax;
}

// grid: any, block 256
__global__ void k_bound_geom(const int32_t* __restrict__ tray, int nx, int ny, int nz, BoundGeom* g) {
    pdl_enter();
    const size_t V = (size_t)nx * ny * nz;
    int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {-1, -1, -1}, h[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) h[k] = INT_MIN;
    bool any = false;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < V; t += (size_t)gridDim.x * blockDim.x) {
        if (tray[t] != 1) continue;
        any = true;
        const size_t r = t / nz;
        const int c[3] = {(int)(r / ny), (int)(r % ny), (int)(t % nz)};
#pragma unroll
        for (int a = 0; a < 3; ++a) { lo[a] = min(lo[a], c[a]); hi[a] = max(hi[a], c[a]); }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            h[k] = max(h[k], ((k & 1) ? -c[0] : c[0]) + ((k & 2) ? -c[1] : c[1]) + ((k & 4) ? -c[2] : c[2]));
    }
    if (!__any_sync(0xffffffffu, any)) return;
    const bool l0 = (threadIdx.x & 31) == 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = __reduce_min_sync(0xffffffffu, lo[a]);
        hi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
        if (l0) { atomicMin(&g->lo[a], lo[a]); atomicMax(&g->hi[a], hi[a]); }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        h[k] = __reduce_max_sync(0xffffffffu, h[k]);
        if (l0) atomicMax(&g->h[k], h[k]);
    }
    if (l0) g->any = 1;
}

// A distance field handed in by the caller need not be the tray's: the
// largest excess of the bounds over it, which the tables then subtract, and the
// range of its values.
// grid: any, block 256
__global__ void k_bound_over(const int32_t* __restrict__ phi, int nx, int ny, int nz, BoundGeom* g) {
    pdl_enter();
    if (!g->any) return;
    const size_t V = (size_t)nx * ny * nz;
    long long over = 0;
    int pmax = 0;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < V; t += (size_t)gridDim.x * blockDim.x) {
        const size_t r = t / nz;
        const int c[3] = {(int)(r / ny), (int)(r % ny), (int)(t % nz)};
        int b = 0;
#pragma unroll
        for (int a = 0; a < 3; ++a) b += max(0, max(g->lo[a] - c[a], c[a] - g->hi[a]));
#pragma unroll
        for (int k = 0; k < 8; ++k)
            b = max(b, ((k & 1) ? -c[0] : c[0]) + ((k & 2) ? -c[1] : c[1]) + ((k & 4) ? -c[2] : c[2]) - g->h[k]);
        const int p = phi[t];
        over = max(over, (long long)b - p);
        pmax = max(pmax, p < 0 ? -1 - p : p);
    }
    const int o = __reduce_max_sync(0xffffffffu, (int)min(over, (long long)INT_MAX));
    pmax = __reduce_max_sync(0xffffffffu, pmax);
    if ((threadIdx.x & 31) != 0) return;
    if (o > 0) atomicMax(&g->over, o);
    atomicMax(&g->pmax, pmax);
}

// ---------------------------------------------------------------------------
// bound tables of one orientation of one item
// ---------------------------------------------------------------------------
// doubles: [0] W, [1..8] s.M - W h(s) per sign vector, [9..11] the numbers of
// x, y, z translations (x: 0 when the orientation is skipped), [12..14] its runs
// (RunHead), [15] the slack of the z cut, infinite where the exact scores
// themselves do not fit (the search then goes to the transforms), then X[nx],
// Y[ny], Z[nz], and the smallest bounded score at z or above of the separable
// bound's z part (F0[nz]) and of W z (F1[nz]), which grow with z, so the last z
// worth testing in a column is a binary search.
// The bounds are integers, exact while they stay below 2^53.  Heavier items
// (values in the millions) pass that: [1..8] and X are then lowered by more than
// every rounding of the sums made of them, so that no bound rounds above its
// score.
struct BoundTab {
    const double *X, *Y, *Z, *F0, *F1;
    const double* c;
    double W;
};
__host__ __device__ inline long long bound_tab_stride(int nx, int ny, int nz) { return PSB_BHDR + nx + ny + 3LL * nz; }

__device__ __forceinline__ BoundTab bound_tab(const double* tab, const ScoreParams& sp) {
    BoundTab b;
    b.W = tab[0];
    b.c = tab + 1;
    b.X = tab + PSB_BHDR;
    b.Y = b.X + sp.nx;
    b.Z = b.Y + sp.ny;
    b.F0 = b.Z + sp.nz;
    b.F1 = b.F0 + sp.nz;
    return b;
}

// Orientations that turn the item into the same array as an earlier one: a
// solid of revolution has 3 different ones of 24, a superellipsoid 6, an
// extruded profile 6 to 12.  Such an orientation's results equal the earlier
// one's, which wins the tie, so it is skipped.  The arrays are compared voxel by
// voxel (a pair that differs mostly does so within the first thousand).
// grid: (n, items), block 256
__global__ void __launch_bounds__(256)
k_bound_dedupe(OrientDesc* __restrict__ od_all, int n) {
    pdl_enter();
    OrientDesc* od = od_all + (size_t)blockIdx.y * n;
    const int o = blockIdx.x;
    const OrientDesc& d = od[o];
    if (d.skip) return;
    const int e0 = d.e[0], e1 = d.e[1], e2 = d.e[2], m = e0 * e1 * e2;
    // source index of oriented (i, j, k): at + i si + j sj + k sk
    auto strides = [](const OrientDesc& q, int* st) {
        const int b[3] = {q.b[1] * q.b[2], q.b[2], 1};
        st[3] = 0;
        for (int a = 0; a < 3; ++a) {
            const int s = q.src_axis[a] == 0 ? b[0] : (q.src_axis[a] == 1 ? b[1] : b[2]);
            st[a] = q.flip[a] ? -s : s;
            if (q.flip[a]) st[3] += (q.e[a] - 1) * s;
        }
    };
    int s1[4], s2[4];
    strides(d, s1);
    const int32_t* v = d.item;
    for (int p = 0; p < o; ++p) {
        const OrientDesc& q = od[p];
        if (q.e[0] != e0 || q.e[1] != e1 || q.e[2] != e2) continue;
        strides(q, s2);
        bool same = true;
        for (int t0 = 0; t0 < m && same; t0 += 1024) {
            bool diff = false;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int t = t0 + 256 * u + threadIdx.x;
                if (t >= m) continue;
                const int k = t % e2, j = t / e2 % e1, i = t / (e2 * e1);
                diff |= __ldg(&v[s1[3] + i * s1[0] + j * s1[1] + k * s1[2]]) !=
                        __ldg(&v[s2[3] + i * s2[0] + j * s2[1] + k * s2[2]]);
            }
            same = !__syncthreads_or(diff);
        }
        if (same) {
            if (threadIdx.x == 0) od[o].skip = 1;
            return;
        }
    }
}

// The tables, and the shift-sorted filter samples (as k_cand_prep), of every
// orientation of the items of a queue: they depend on the items and the sources
// only, so one launch serves them all.
// grid: (n, items), block 256
template <int NW>
__global__ void __launch_bounds__(256)
k_bound_prep(const OrientDesc* __restrict__ od_all, int n, const BoundGeom* __restrict__ geom, ScoreParams sp,
             double* __restrict__ tab, long long tstride, int2* __restrict__ fs, int* __restrict__ fbound) {
    pdl_enter();
    // marginals, their prefix sums and the prefix sums of k times them
    __shared__ unsigned long long hm[3][PSB_MAX_FFT + 1], c0[3][PSB_MAX_FFT + 1], c1[3][PSB_MAX_FFT + 1];
    __shared__ double sM[3], sW;
    const int slot = blockIdx.y * n + blockIdx.x;
    const OrientDesc& od = od_all[slot];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double* T = tab + (size_t)slot * tstride;
    if (tid < 3) T[9 + tid] = od.skip ? 0.0 : (double)od.valid[tid];
    if (od.skip) return;
    if (tid == 3) {
        const bool ax = od.src_axis[0] == (od.src_axis[2] == 0 ? 1 : 0);   // the tray's x comes from a run's q.x
        T[12] = (double)od.nruns;
        T[13] = __longlong_as_double((long long)od.runs);
        T[14] = __longlong_as_double((long long)od.e[0] | (long long)od.e[1] << 12 | (long long)od.e[2] << 24 |
                                     (long long)(od.flip[0] != 0) << 36 | (long long)(od.flip[1] != 0) << 37 |
                                     (long long)(od.flip[2] != 0) << 38 | (long long)ax << 39);
    }
    // marginals of the oriented item along x, y and z (z by differences)
    for (int i = tid; i < 3 * (PSB_MAX_FFT + 1); i += 256) (&hm[0][0])[i] = 0ULL;
    __syncthreads();
    for (int r = tid; r < od.nruns; r += 256) {
        const int4 q = __ldg(&od.runs[r]);
        int a, b, z0, z1;
        orient_run(od, q, &a, &b, &z0, &z1);
        const unsigned long long w = (unsigned long long)(long long)q.w, wl = w * (unsigned long long)(z1 - z0 + 1);
        atomicAdd(&hm[0][a], wl);
        atomicAdd(&hm[1][b], wl);
        atomicAdd(&hm[2][z0], w);
        atomicAdd(&hm[2][z1 + 1], 0ULL - w);
    }
    __syncthreads();
    if (warp == 0) {
        unsigned long long carry = 0;
        for (int k0 = 0; k0 < od.e[2]; k0 += 32) {
            unsigned long long v = k0 + lane < od.e[2] ? hm[2][k0 + lane] : 0ULL;
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned long long u = __shfl_up_sync(0xffffffffu, v, d);
                if (lane >= d) v += u;
            }
            v += carry;
            if (k0 + lane < od.e[2]) hm[2][k0 + lane] = v;
            carry = __shfl_sync(0xffffffffu, v, 31);
        }
    }
    __syncthreads();
    if (warp < 3) {
        unsigned long long w = 0, m = 0;
        const int e = od.e[warp];
        if (lane == 0) c0[warp][0] = c1[warp][0] = 0ULL;
        for (int k0 = 0; k0 < e; k0 += 32) {
            unsigned long long v = k0 + lane < e ? hm[warp][k0 + lane] : 0ULL, u = v * (unsigned long long)(k0 + lane);
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned long long v2 = __shfl_up_sync(0xffffffffu, v, d);
                const unsigned long long u2 = __shfl_up_sync(0xffffffffu, u, d);
                if (lane >= d) { v += v2; u += u2; }
            }
            v += w;
            u += m;
            if (k0 + lane < e) { c0[warp][k0 + lane + 1] = v; c1[warp][k0 + lane + 1] = u; }
            w = __shfl_sync(0xffffffffu, v, 31);
            m = __shfl_sync(0xffffffffu, u, 31);
        }
        if (lane == 0) {
            sM[warp] = (double)m;
            if (warp == 0) sW = (double)w;
        }
    }
    __syncthreads();
    // no part or sum of a bound exceeds top; a sum is a dozen operations at
    // most, each off by 2^-53 of that
    const double W = sW, top = W * ((double)geom->over + 8.0 * (sp.nx + sp.ny + sp.nz));
    const double low = -W * (double)geom->over - (top < 9007199254740992.0 ? 0.0 : 0x1p-49 * top);
    if (tid == 0) {
        T[0] = W;
        // a run's proximity (up to 256 cells) is a 32-bit sum, an item's and its
        // moments (k times the weights) 64-bit ones
        const double pmax = geom->pmax;
        T[15] = pmax < 8388608.0 && W * fmax(pmax + 1.0, 1024.0) < 0x1p62 ? 1e-6 + 1e-15 * top : INFINITY;
    }
    if (tid < 8)
        T[1 + tid] = ((tid & 1) ? -sM[0] : sM[0]) + ((tid & 2) ? -sM[1] : sM[1]) + ((tid & 4) ? -sM[2] : sM[2]) -
                     W * (double)geom->h[tid] + low;
    double* part[3] = {T + PSB_BHDR, T + PSB_BHDR + sp.nx, T + PSB_BHDR + sp.nx + sp.ny};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        // sum over k of hm[k] max(0, lo - p - k, p + k - hi): the cells before
        // the box are k < m1, those behind it k >= m2
        const long long lo = geom->lo[a], hi = geom->hi[a], e = od.e[a];
        for (int p = tid; p < od.valid[a]; p += 256) {
            const long long m1 = min(max(lo - p, 0LL), e), m2 = min(max(hi - p + 1, 0LL), e);
            const long long v = (lo - p) * (long long)c0[a][m1] - (long long)c1[a][m1] +
                                (p - hi) * (long long)(c0[a][e] - c0[a][m2]) + (long long)(c1[a][e] - c1[a][m2]);
            part[a][p] = (double)v + (a == 0 ? low : 0.0);
        }
    }
    __syncthreads();
    if (warp < 2) {
        // smallest bounded score at z or above
        const double* Z = part[2];
        double* F = part[2] + (warp == 0 ? sp.nz : 2 * sp.nz);
        double carry = INFINITY;
        const int Zv = od.valid[2];
        for (int z0 = ((Zv - 1) / 32) * 32; z0 >= 0 && Zv > 0; z0 -= 32) {
            const int z = z0 + lane;
            double v = INFINITY;
            if (z < Zv) v = (warp == 0 ? Z[z] : W * (double)z) + ref_score(sp, 0.0, z);
            for (int d = 1; d < 32; d <<= 1) {
                const double u = __shfl_down_sync(0xffffffffu, v, d);
                if (lane + d < 32) v = fmin(v, u);
            }
            v = fmin(v, carry);
            if (z < Zv) F[z] = v;
            carry = __shfl_sync(0xffffffffu, v, 0);
        }
    }
    if (warp == 2) {
        // the buckets padded to whole batches with copies of their first
        // sample, so the filter needs no test per sample
        __shared__ int sb[PSB_FBOUND];
        __shared__ int2 ss[PSB_FSAMP];
        sort_samples<NW>(od, sb, lane, [&](int i, int x, int y, int z) {
            ss[i] = make_int2((x * sp.ny + y) * (NW / 4), z & 31);
        });
        __syncwarp();
        int2* S = fs + (size_t)slot * PSB_BSAMP;
        int base = 0;
        for (int k = 0; k < NW; ++k) {
            const int b0 = sb[k], m = sb[k + 1] - b0, p = (m + PSB_BBATCH - 1) / PSB_BBATCH * PSB_BBATCH;
            if (lane == 0) fbound[(size_t)slot * PSB_FBOUND + k] = base;
            for (int i = lane; i < p; i += 32) S[base + i] = ss[b0 + (i < m ? i : 0)];
            base += p;
        }
        if (lane == 0) fbound[(size_t)slot * PSB_FBOUND + NW] = base;
    }
}

// ---------------------------------------------------------------------------
// exact checks of one translation, by one warp over the item's z-runs
// ---------------------------------------------------------------------------
// A run meets an occupied cell when one of the free bits of its tray column
// over its z range is clear (one or two words for most runs).
__device__ __forceinline__ bool run_blocked(const uint32_t* __restrict__ col, int z0, int z1) {
    const int w0 = z0 >> 5, w1 = z1 >> 5;
    const uint32_t m0 = 0xffffffffu << (z0 & 31), m1 = 0xffffffffu >> (31 - (z1 & 31));
    if (w0 == w1) return (~__ldg(&col[w0]) & m0 & m1) != 0u;
    uint32_t bad = (~__ldg(&col[w0]) & m0) | (~__ldg(&col[w1]) & m1);
    for (int w = w0 + 1; w < w1; ++w) bad |= ~__ldg(&col[w]);
    return bad != 0u;
}

// An orientation's runs, from its table's header (entry l in lane l), so that
// a check starts without another round trip for the descriptor.
struct RunHead {
    const int4* runs;
    int nr;
    long long code;             // extents, flips and the axis of q.x
};
__device__ __forceinline__ RunHead run_head(double h) {
    RunHead r;
    r.nr = (int)__shfl_sync(0xffffffffu, h, 12);
    r.runs = (const int4*)__double_as_longlong(__shfl_sync(0xffffffffu, h, 13));
    r.code = __double_as_longlong(__shfl_sync(0xffffffffu, h, 14));
    return r;
}
// The map of an item's runs to tray columns and z ranges at a translation:
// orient_run, with everything that does not depend on the run taken out.
struct RunMap {
    int col, mx, my;            // column = col + mx * q.x + my * q.y
    int z;                      // z range = z + c0 .. z + c1
    int ez;                     // flipped: c0 = ez - r1, c1 = ez - r0
    bool flip;
};
__device__ __forceinline__ RunMap run_map(const RunHead& h, int ny, int x, int y, int z) {
    const int e0 = (int)(h.code & 4095), e1 = (int)(h.code >> 12 & 4095);
    const bool f0 = h.code >> 36 & 1, f1 = h.code >> 37 & 1, ax = h.code >> 39 & 1;
    const int sa = f0 ? -ny : ny, sb = f1 ? -1 : 1;
    RunMap m;
    m.mx = ax ? sa : sb;
    m.my = ax ? sb : sa;
    m.col = (x + (f0 ? e0 - 1 : 0)) * ny + y + (f1 ? e1 - 1 : 0);
    m.z = z;
    m.ez = (int)(h.code >> 24 & 4095) - 1;
    m.flip = h.code >> 38 & 1;
    return m;
}
__device__ __forceinline__ int run_at(const RunMap& m, int4 q, int* z0, int* z1) {
    const int r0 = q.z & 0xffff, r1 = q.z >> 16;
    *z0 = m.z + (m.flip ? m.ez - r1 : r0);
    *z1 = m.z + (m.flip ? m.ez - r0 : r1);
    return m.col + m.mx * q.x + m.my * q.y;
}

// Collision-free?  (Item values are positive: negative ones are refused.)
// Each step checks 128 runs spread over the whole item, so a blocked
// translation is mostly found out in the first one.
__device__ __forceinline__ bool bound_free(const RunHead& od, const uint32_t* __restrict__ T, int tw, int ny, int x,
                                           int y, int z) {
    const int lane = threadIdx.x & 31, nr = od.nr, steps = (nr + 127) / 128;
    const int4* runs = od.runs;
    const RunMap rm = run_map(od, ny, x, y, z);
    int4 q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int r = steps * (32 * u + lane);
        q[u] = r < nr ? __ldg(&runs[r]) : make_int4(0, 0, 0, 0);   // values are positive: w = 0 marks none
    }
    for (int i = 0; i < steps; ++i) {
        int4 next[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int r = i + 1 + steps * (32 * u + lane);
            next[u] = i + 1 < steps && r < nr ? __ldg(&runs[r]) : make_int4(0, 0, 0, 0);
        }
        bool hit = false;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (q[u].w == 0) continue;
            int z0, z1;
            const int col = run_at(rm, q[u], &z0, &z1);
            hit = run_blocked(T + (size_t)col * tw, z0, z1) || hit;
        }
        if (__any_sync(0xffffffffu, hit)) return false;
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = next[u];
    }
    return true;
}

// Exact proximity (every lane returns it), from the distance field's prefix
// sums along z.
__device__ __forceinline__ long long bound_prox(const RunHead& od, const int32_t* __restrict__ pphi, int ny, int nz,
                                                int x, int y, int z) {
    const int lane = threadIdx.x & 31, nr = od.nr;
    const int4* runs = od.runs;
    const RunMap rm = run_map(od, ny, x, y, z);
    long long acc = 0;
#pragma unroll 4
    for (int r = lane; r < nr; r += 32) {
        const int4 q = __ldg(&runs[r]);
        int z0, z1;
        const int32_t* P = pphi + (size_t)run_at(rm, q, &z0, &z1) * (nz + 1);
        acc += (long long)q.w * (__ldg(&P[z1 + 1]) - __ldg(&P[z0]));
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    return acc;
}

// The best score and the count as they are now.  Other warps are changing them,
// so one lane reads for the warp: lanes that each read for themselves could see
// different values and part ways around a warp-wide vote.  (Called by whole warps.)
__device__ __forceinline__ double bound_best(const BoundState* st) {
    unsigned long long k = 0ULL;
    if ((threadIdx.x & 31) == 0) k = *(const volatile unsigned long long*)&st->best;
    k = __shfl_sync(0xffffffffu, k, 0);
    return k == 0xffffffffffffffffULL ? INFINITY : ord_val(k);
}
// both in one load; returns the best score
__device__ __forceinline__ double bound_now(const BoundState* st, int* listed) {
    int4 a = make_int4(0, 0, 0, 0);
    if ((threadIdx.x & 31) == 0) a = __ldcg((const int4*)st);
    *listed = __shfl_sync(0xffffffffu, a.z, 0);
    const unsigned int lo = __shfl_sync(0xffffffffu, a.x, 0), hi = __shfl_sync(0xffffffffu, a.y, 0);
    const unsigned long long k = lo | (unsigned long long)hi << 32;
    return k == 0xffffffffffffffffULL ? INFINITY : ord_val(k);
}

// largest octant bound of a column for z signs + (gp, add W z) and - (gm)
__device__ __forceinline__ void bound_octants(const BoundTab& b, int x, int y, double* gp, double* gm) {
    const double dx = b.W * (double)x, dy = b.W * (double)y;
    *gp = fmax(fmax(dx + dy + b.c[0], -dx + dy + b.c[1]), fmax(dx - dy + b.c[2], -dx - dy + b.c[3]));
    *gm = fmax(fmax(dx + dy + b.c[4], -dx + dy + b.c[5]), fmax(dx - dy + b.c[6], -dx - dy + b.c[7]));
}

// the runs of orientation o (a warp-wide load of its header)
__device__ __forceinline__ RunHead run_head_of(const double* __restrict__ tab, long long tstride, int o) {
    return run_head(tab[(size_t)o * tstride + min((int)(threadIdx.x & 31), 14)]);
}

// the bounded score of cell z of a column (A = X + Y, octant parts gp, gm)
__device__ __forceinline__ double bound_score(const BoundTab& b, const ScoreParams& sp, double A, double gp, double gm,
                                              int z) {
    const double wz = b.W * (double)z;
    return ref_score(sp, fmax(A + b.Z[z], fmax(gp + wz, gm - wz)), z);
}

// how many of the nondecreasing F[0..n) are <= lim
__device__ __forceinline__ int bound_count(const double* __restrict__ F, int n, double lim) {
    int lo = 0;
    while (lo < n) {
        const int mid = (lo + n) >> 1;
        if (F[mid] <= lim) lo = mid + 1;
        else n = mid;
    }
    return lo;
}

struct BoundArgs {
    BoundState* st;
    const double* tab;          // the item's tables (orientation stride tstride)
    long long tstride;
    const int2* fs;             // its samples: column offset, bit shift (PSB_BSAMP per orientation)
    const int* fbound;
    BoundHit* list;
    BoundHit* win;
    const int32_t* pphi;
};

// The sample filter on 32 columns of translations (lane = one y, col its
// tray column): c, handed in with the z range to test, is ANDed with the
// tray's free bits of column (x + s.x, y + s.y) shifted down by s.z for every
// sample s; the warp stops once no lane holds a survivor.  Only the lowest WA
// words of c are live: with the z range cut by the bounds that is mostly one
// or two, and a sample then costs its two loads and two instructions per
// live word (128 samples by themselves are most of a warp's instructions: with
// all words, tests per sample and samples handed round by shuffles, 4.3 M per
// seed pass at 128^3 and 24 orientations, a warp's chain 38k cycles long).
// Batches first, first + step, ... of each bucket are taken.
template <int NQ, int WA, int BATCH>
__device__ __forceinline__ void bound_filter(const uint4* __restrict__ col, const int2* __restrict__ fs, int fb,
                                             int first, int step, uint32_t (&c)[4 * NQ]) {
    constexpr int NW = 4 * NQ;
#pragma unroll
    for (int k = 0; k < NW; ++k) {
        // the quads holding words k .. k + WA of a column
        constexpr int NQ1 = NQ;
        const int u0 = k / 4, u1 = (k + WA) / 4 < NQ1 ? (k + WA) / 4 : NQ1 - 1;
        const int s1 = __shfl_sync(0xffffffffu, fb, k + 1);
        for (int s0 = __shfl_sync(0xffffffffu, fb, k) + first * BATCH; s0 < s1; s0 += step * BATCH) {
            uint32_t a = 0u;
#pragma unroll
            for (int w = 0; w < WA; ++w) a |= c[w];
            if (!__any_sync(0xffffffffu, a != 0u)) return;
            uint4 v[BATCH][NQ];
            int off[BATCH];
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                const int2 q = __ldg(&fs[s0 + i]);
                off[i] = q.y;
#pragma unroll
                for (int u = 0; u < NQ; ++u)
                    v[i][u] = u >= u0 && u <= u1 ? __ldg(col + q.x + u) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                uint32_t T[NW + 1];
#pragma unroll
                for (int u = 0; u < NQ; ++u) {
                    T[4 * u] = v[i][u].x;
                    T[4 * u + 1] = v[i][u].y;
                    T[4 * u + 2] = v[i][u].z;
                    T[4 * u + 3] = v[i][u].w;
                }
                T[NW] = 0u;
#pragma unroll
                for (int w = 0; w < WA; ++w) {
                    const uint32_t lo = (w + k < NW) ? T[w + k] : 0u;
                    const uint32_t hi = (w + k + 1 < NW) ? T[w + k + 1] : 0u;
                    c[w] &= __funnelshift_r(lo, hi, off[i]);
                }
            }
        }
    }
}

// What a pass needs of 32 columns: the orientation's table, the columns'
// parts of the bounds (lane = column) and the z range worth testing.
struct BoundCols {
    BoundTab bt;
    int fb;                     // sample bucket bounds, one per lane
    double h;                   // the table's header, one entry per lane
    int Yv;
    bool any;                   // a column has a z range
    double A, gp, gm;
    int zc;
};
// lane's row y of plane x; best: INFINITY for the whole range
__device__ __forceinline__ BoundCols bound_cols(const BoundArgs& ba, const ScoreParams& sp, int nw, int o, int x, int y,
                                                double best) {
    const int lane = threadIdx.x & 31;
    BoundCols c;
    c.bt = bound_tab(ba.tab + (size_t)o * ba.tstride, sp);
    const double h = c.h = c.bt.c[min(lane, 15) - 1];   // lane l: header entry l
    c.fb = lane <= nw ? __ldg(&ba.fbound[(size_t)o * PSB_FBOUND + lane]) : 0;
    const int Xv = (int)__shfl_sync(0xffffffffu, h, 9), Zv = (int)__shfl_sync(0xffffffffu, h, 11);
    c.Yv = (int)__shfl_sync(0xffffffffu, h, 10);
    const bool act = x < Xv && y < c.Yv;
    c.A = c.gp = c.gm = 0.0;
    c.zc = act ? Zv : 0;
    if (act) {
        c.A = c.bt.X[x] + c.bt.Y[y];
        bound_octants(c.bt, x, y, &c.gp, &c.gm);
    }
    if (best < INFINITY) {
        // slack for the roundings of F's sums; the exact test follows
        const double lim = best + 1e-12 * fabs(best) + __shfl_sync(0xffffffffu, h, 15);
        if (!act || c.bt.F0[0] > lim - c.A || c.bt.F1[0] > lim - c.gp) c.zc = 0;
        if (__any_sync(0xffffffffu, c.zc > 0) && c.zc > 0) {
            c.zc = bound_count(c.bt.F0, Zv, lim - c.A);
            c.zc = bound_count(c.bt.F1, c.zc, lim - c.gp);
        }
    }
    c.any = __any_sync(0xffffffffu, c.zc > 0);
    return c;
}

// The tasks of a pass: planes x row blocks of the orientations that are searched
// (of at most 32, those the tables do not mark skipped; a skipped one's tasks
// would each cost a round trip for its header).
struct BoundTasks {
    unsigned int mask;
    int n, planes, yb, count;
    __device__ __forceinline__ int orient(int k) const { return n <= 32 ? (int)__fns(mask, 0, k + 1) : k; }
};
__device__ __forceinline__ BoundTasks bound_tasks(const BoundArgs& ba, const ScoreParams& sp, int n, int xstep, int rows) {
    BoundTasks t;
    t.n = n;
    const int lane = threadIdx.x & 31;
    int m = n, X = sp.nx, Y = sp.ny;
    t.mask = ~0u;
    if (n <= 32) {
        const double* h = ba.tab + (size_t)min(lane, n - 1) * ba.tstride;
        const int xv = lane < n ? (int)h[9] : 0;
        t.mask = __ballot_sync(0xffffffffu, xv > 0);
        m = __popc(t.mask);
        X = __reduce_max_sync(0xffffffffu, xv);
        Y = __reduce_max_sync(0xffffffffu, xv > 0 ? (int)h[10] : 0);
    }
    t.planes = (X + xstep - 1) / xstep;
    t.yb = (Y + rows - 1) / rows;
    t.count = m * t.planes * t.yb;
    return t;
}

// The first pass: a best score to cut the second one with, from a lattice of
// columns (every fourth plane, the first four of every 16 rows: rows one by
// one would touch a cache line each).  There are few tasks and each is a
// chain of load latencies, so a CTA takes one: its four warps share the
// samples, meet in shared memory, and then check and score the four survivors
// of lowest bound, one each.  Bound by those latencies: 13 % of the cycles issue,
// 8.6 of 14.2 cycles per instruction wait for a load (a 128^3 tray, 24
// orientations: 744 CTAs, 20 us).  So the CTAs per SM matter little: 6 (80
// registers, 100 bytes spilled) and 4 (128 registers, 12 bytes) give 1.44 and
// 1.45 ms for 20 boxes at 64^3, 7.9 and 8.1 ms for 100 items at 128^3, 42.2 and
// 41.5 ms for 350 at 240x123x100, where runs of one side differ by up to 8 %.
// grid: any, block 128
template <int NQ>
__global__ void __launch_bounds__(128, NQ == 1 ? 6 : 3)
k_bound_seed(int n, const uint4* __restrict__ tbits, ScoreParams sp,
             BoundArgs ba) {
    pdl_enter();
    constexpr int NW = 4 * NQ;
    __shared__ uint32_t cs[4][NW][32];
    BoundState* st = ba.st;
    if (bound_entry(st).halt) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ny = sp.ny;
    const BoundTasks tm = bound_tasks(ba, sp, n, PSB_BSTEP, 128);
    for (int task = blockIdx.x; task < tm.count; task += gridDim.x) {
        const int y0 = task % tm.yb * 128, yl = y0 + lane / 4 * 16 + lane % 4;
        const int x = task / tm.yb % tm.planes * PSB_BSTEP, o = tm.orient(task / (tm.yb * tm.planes));
        // (the same in all four warps but for the best score, so no early exit on it)
        const BoundCols bc = bound_cols(ba, sp, NW, o, x, yl, INFINITY);
        if (!bc.any) continue;
        uint32_t c[NW];
#pragma unroll
        for (int w = 0; w < NW; ++w) c[w] = low_bits(bc.zc - 32 * w);
        const uint4* col = tbits + ((size_t)x * ny + min(yl, bc.Yv - 1)) * NQ;
        bound_filter<NQ, NW, PSB_BBATCH / NQ>(col, ba.fs + (size_t)o * PSB_BSAMP, bc.fb, warp, 4, c);
        __syncthreads();   // the last task's survivors have been read
#pragma unroll
        for (int w = 0; w < NW; ++w) cs[warp][w][lane] = c[w];
        __syncthreads();
#pragma unroll
        for (int w = 0; w < NW; ++w) c[w] = cs[0][w][lane] & cs[1][w][lane] & cs[2][w][lane] & cs[3][w][lane];
        // this warp's survivor: the warp-th lowest bounded score among the
        // first survivors of each word
        const double now = bound_best(st);
        double lb[NW];
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            lb[w] = INFINITY;
            if (c[w]) lb[w] = bound_score(bc.bt, sp, bc.A, bc.gp, bc.gm, 32 * w + __ffs(c[w]) - 1);
        }
        double m = INFINITY;
        int src = 0, zz = -1;
        for (int k = 0; k <= warp; ++k) {
            double own = INFINITY;
            int lw = -1;
#pragma unroll
            for (int w = 0; w < NW; ++w)
                if (lb[w] < own) { own = lb[w]; lw = w; }
            m = own;
            for (int d = 16; d > 0; d >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, d));
            const unsigned int who = __ballot_sync(0xffffffffu, lw >= 0 && own == m);
            zz = -1;
            if (!who) break;
            src = __ffs(who) - 1;
            int z = -1;
#pragma unroll
            for (int w = 0; w < NW; ++w)
                if (w == lw) {
                    z = 32 * w + __ffs(c[w]) - 1;
                    if (lane == src) lb[w] = INFINITY;
                }
            zz = __shfl_sync(0xffffffffu, z, src);
        }
        if (zz < 0 || !(m < now)) continue;
        const RunHead od = run_head(bc.h);
        const int y = y0 + src / 4 * 16 + src % 4;
        if (!bound_free(od, (const uint32_t*)tbits, NW, ny, x, y, zz)) continue;
        const long long D = bound_prox(od, ba.pphi, ny, sp.nz, x, y, zz);
        if (lane == 0) atomicMin(&st->best, ord_key(ref_score(sp, (double)D, zz)));
    }
}

// The second pass: one warp takes 32 columns (x, y0 + lane) of one orientation
// at a time; the grid is sized to the chip and strides over the tasks (a CTA
// per plane and orientation spent its time starting: 5,760 short CTAs per item
// at 240x123x100), orientations outermost, so that the warps of an SM share a
// few tables.  ALL: every survivor for the flood, whatever its score (gated).
// grid: any, block 128
template <int NQ, bool ALL>
__global__ void __launch_bounds__(128, NQ == 1 ? 6 : 4)
k_bound_find(int n, const uint4* __restrict__ tbits, ScoreParams sp,
             BoundArgs ba) {
    pdl_enter();
    BoundState* st = ba.st;
    const BoundEntry en = bound_entry(st);
    if (en.halt || (ALL && !en.need_flood)) return;
    constexpr int NW = 4 * NQ;
    constexpr int BATCH = 8 / NQ;
    const int lane = threadIdx.x & 31, ny = sp.ny;
    const BoundTasks tm = bound_tasks(ba, sp, n, 1, 32);
    const int nwarps = gridDim.x * (blockDim.x >> 5);
    for (int task = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); task < tm.count; task += nwarps) {
        const int y0 = task % tm.yb * 32, x = task / tm.yb % tm.planes, o = tm.orient(task / (tm.yb * tm.planes));
        int listed;
        double best = bound_now(st, &listed);
        if (ALL) best = INFINITY;
        if (listed > PSB_BCAP) return;   // the list is lost anyway
        const BoundCols bc = bound_cols(ba, sp, NW, o, x, y0 + lane, best);
        if (!(__shfl_sync(0xffffffffu, bc.h, 15) < INFINITY)) {   // not scored here: the list counts as lost
            if (lane == 0) atomicMax(&st->count, PSB_BCAP + 1);
            return;
        }
        if (!bc.any) continue;
        const BoundTab& bt = bc.bt;
        const double A = bc.A, gp = bc.gp, gm = bc.gm;
        const int y = y0 + lane;
        uint32_t c[NW];
        uint32_t some = 0u;
#pragma unroll
        for (int w = 0; w < NW; ++w) c[w] = low_bits(bc.zc - 32 * w);
        // (a lane past the last row reads the last one's columns)
        const uint4* col = tbits + ((size_t)x * ny + min(y, bc.Yv - 1)) * NQ;
        const int2* fs = ba.fs + (size_t)o * PSB_BSAMP;
        const int top = __reduce_max_sync(0xffffffffu, bc.zc), fb = bc.fb;
        if (top <= 32) bound_filter<NQ, 1, BATCH>(col, fs, fb, 0, 1, c);
        else if (top <= 64) bound_filter<NQ, 2, BATCH>(col, fs, fb, 0, 1, c);
        else bound_filter<NQ, NW, BATCH>(col, fs, fb, 0, 1, c);
#pragma unroll
        for (int w = 0; w < NW; ++w) some |= c[w];
        if (!__any_sync(0xffffffffu, some != 0u)) continue;
        int held = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) held += __popc(c[w]);
        held = __reduce_add_sync(0xffffffffu, held);
        if (!ALL && (held > 32 || !(best < INFINITY))) {
            // no seed found a free translation, or a loose one: try this warp's
            // best before listing them all
            const RunHead od = run_head(bc.h);
            for (int tries = 0; tries < 3; ++tries) {
                // the lowest bounded score among the first survivors of each word
                double lb = INFINITY;
                int lz = -1;
#pragma unroll
                for (int w = 0; w < NW; ++w)
                    if (c[w]) {
                        const int z = 32 * w + __ffs(c[w]) - 1;
                        const double s = bound_score(bt, sp, A, gp, gm, z);
                        if (s < lb) { lb = s; lz = z; }
                    }
                double m = lb;
                for (int d = 16; d > 0; d >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, d));
                if (!(m < bound_best(st))) break;   // no survivor, or none that could improve
                const int src = __ffs(__ballot_sync(0xffffffffu, lz >= 0 && lb == m)) - 1;
                const int zz = __shfl_sync(0xffffffffu, lz, src);
                if (bound_free(od, (const uint32_t*)tbits, NW, ny, x, y0 + src, zz)) {
                    const long long D = bound_prox(od, ba.pphi, ny, sp.nz, x, y0 + src, zz);
                    if (lane == 0) atomicMin(&st->best, ord_key(ref_score(sp, (double)D, zz)));
                    break;
                }
#pragma unroll
                for (int w = 0; w < NW; ++w)   // blocked: no survivor
                    if (lane == src && (zz >> 5) == w) c[w] &= ~(1u << (zz & 31));
            }
            best = bound_best(st);
        }
        int mine = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            if (best < INFINITY) {
                for (uint32_t m = c[w]; m; m &= m - 1u) {
                    const int z = 32 * w + __ffs(m) - 1;
                    if (bound_score(bt, sp, A, gp, gm, z) > best) c[w] &= ~(1u << (z & 31));
                }
            }
            mine += __popc(c[w]);
        }
        int incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += u;
        }
        int slot = 0;
        if (lane == 31 && incl) slot = atomicAdd(&st->count, incl);
        slot = __shfl_sync(0xffffffffu, slot, 31) + incl - mine;
#pragma unroll
        for (int w = 0; w < NW; ++w)
            for (uint32_t m = c[w]; m && slot < PSB_BCAP; m &= m - 1u, ++slot) {
                const int z = 32 * w + __ffs(m) - 1;
                BoundHit h2;
                h2.t = (x * ny + y) * sp.nz + z;
                h2.o = o;
                h2.s = bound_score(bt, sp, A, gp, gm, z);
                ba.list[slot] = h2;
            }
    }
}

// The item's outcome into the loop state and its decision record
__device__ __forceinline__ void bound_commit(LoopState* ls, DecisionDev* out, const ScoreParams& sp, int o, int t,
                                             double s, int ncand, bool flood = false) {
    DecisionDev d;
    // decided without transforms; by a second selection after the flood fill
    d.diag = flood ? 0xc00u : 0x800u;
    d.ncand = ncand;
    d.err_ratio = 0.f;
    d.found = o >= 0;
    d.orientation = o;
    d.score = o >= 0 ? s : 0.0;
    d.x = o >= 0 ? t / (sp.nz * sp.ny) : -1;
    d.y = o >= 0 ? (t / sp.nz) % sp.ny : -1;
    d.z = o >= 0 ? t % sp.nz : -1;
    *out = d;
    ls->do_place = d.found;
    if (!d.found) return;
    ls->orient = o;
    ls->px = d.x; ls->py = d.y; ls->pz = d.z;
    ls->id = ls->id_offset + ls->placed + 1;
    ls->placed += 1;
}

// Exact check and score of the listed translations, one warp each, then the
// winner (in the last CTA to finish): smallest score, on equal scores the
// lowest orientation, then the tie key within it.  FLOOD: the second pass,
// over the translations k_bound_flood left (free and reachable, the others
// carry 1e300).  grid: any, block 256
template <bool FLOOD>
__global__ void __launch_bounds__(256)
k_bound_score(const uint4* __restrict__ tbits, int tq, ScoreParams sp, BoundArgs ba, int item, int interlock,
              LoopState* ls, DecisionDev* out) {
    pdl_enter();
    BoundState* st = ba.st;
    const BoundEntry en = bound_entry(st);
    if (en.halt || (FLOOD && !en.need_flood)) return;
    const int count = en.count;
    const bool fail = count > PSB_BCAP;
    const int n = fail ? 0 : count;
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    __shared__ long long part[8];
    auto scored = [&](int t, int o, int z, long long D) {
        const double s = ref_score(sp, (double)D, z);
        if (ord_key(s) <= atomicMin(&st->best, ord_key(s))) {
            // the best so far, or equal to it: a candidate for the tie rules
            BoundHit w;
            w.t = t;
            w.o = o;
            w.s = s;
            ba.win[atomicAdd(&st->nwin, 1)] = w;
        }
    };
    if (n <= (int)gridDim.x) {
        // few entries: a CTA each, every run's loads in flight at once
        for (int e = blockIdx.x; e < n; e += gridDim.x) {
            const BoundHit h = ba.list[e];
            if (!(h.s < 1e299)) continue;
            const RunHead od = run_head_of(ba.tab, ba.tstride, h.o);
            const int z = h.t % sp.nz, y = (h.t / sp.nz) % sp.ny, x = h.t / (sp.nz * sp.ny);
            const RunMap rm = run_map(od, sp.ny, x, y, z);
            const uint32_t* T = (const uint32_t*)tbits;
            long long acc = 0;
            bool hit = false;
#pragma unroll 4
            for (int r = threadIdx.x; r < od.nr; r += 256) {
                const int4 q = __ldg(&od.runs[r]);
                int z0, z1;
                const int col = run_at(rm, q, &z0, &z1);
                const int32_t* P = ba.pphi + (size_t)col * (sp.nz + 1);
                acc += (long long)q.w * (__ldg(&P[z1 + 1]) - __ldg(&P[z0]));
                if (!FLOOD) hit = run_blocked(T + (size_t)col * 4 * tq, z0, z1) || hit;
            }
            for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
            if (lane == 0) part[threadIdx.x >> 5] = acc;
            if (__syncthreads_or(hit)) continue;
            if (threadIdx.x == 0) {
                for (int k = 1; k < wpb; ++k) acc += part[k];
                scored(h.t, h.o, z, acc);
            }
            __syncthreads();
        }
    }
    // many: two per warp and step, most found blocked by their first 128 runs
    for (int e0 = n <= (int)gridDim.x ? n : 2 * (blockIdx.x * wpb + (threadIdx.x >> 5)); e0 < n;
         e0 += 2 * gridDim.x * wpb) {
        BoundHit h;
        h.t = h.o = 0;
        h.s = 1e300;
        if (lane < 2 && e0 + lane < n) h = ba.list[e0 + lane];
        for (unsigned int m = __ballot_sync(0xffffffffu, h.s < 1e299); m; m &= m - 1u) {
            const int src = __ffs(m) - 1;
            const int t = __shfl_sync(0xffffffffu, h.t, src), o = __shfl_sync(0xffffffffu, h.o, src);
            if (__shfl_sync(0xffffffffu, h.s, src) > bound_best(st)) continue;
            const RunHead od = run_head_of(ba.tab, ba.tstride, o);
            const int z = t % sp.nz, y = (t / sp.nz) % sp.ny, x = t / (sp.nz * sp.ny);
            if (!FLOOD && !bound_free(od, (const uint32_t*)tbits, 4 * tq, sp.ny, x, y, z)) continue;
            const long long D = bound_prox(od, ba.pphi, sp.ny, sp.nz, x, y, z);
            if (lane == 0) scored(t, o, z, D);
        }
    }
    __shared__ bool last;
    __shared__ unsigned long long red[8];
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicInc(&st->done, gridDim.x - 1) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    const BoundEntry fin = bound_entry(st);
    const double best = fin.best;
    unsigned long long win = ~0ULL;
    for (int e = threadIdx.x; e < fin.nwin; e += blockDim.x) {
        const volatile BoundHit* h = &ba.win[e];
        if (h->s == best)
            win = min(win, ((unsigned long long)(unsigned int)h->o << 32) | tie_key(sp.mode, h->t));
    }
    for (int d = 16; d > 0; d >>= 1) win = min(win, __shfl_xor_sync(0xffffffffu, win, d));
    if (lane == 0) red[threadIdx.x >> 5] = win;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int k = 1; k < wpb; ++k) win = min(win, red[k]);
    st->count = st->nwin = 0;
    st->best = 0xffffffffffffffffULL;
    if (FLOOD) st->need_flood = 0;
    const bool found = best < (sp.mode == 0 ? 1000000000.0 : 1e29);
    if (fail || (found && win == ~0ULL)) {   // (the second cannot be: a score has its translation)
        st->halt = 1;
        st->halt_item = item;
        ls->do_place = 0;
        return;
    }
    const int o = found ? (int)(win >> 32) : -1;
    const int t = found ? untie_key(sp.mode, (unsigned int)win) : -1;
    if (found && interlock && !FLOOD) {
        st->need_ray = 1;
        st->win_o = o;
        st->win_t = t;
        st->win_s = best;
        ls->do_place = 0;
        out->ncand = count;
        return;
    }
    bound_commit(ls, out, sp, o, t, best, count, FLOOD);
}

// Interlocking mode: the cells between the winner and the six faces, one
// warp each (a cell is free when the item fits there, checked exactly); a
// direction without a blocked cell proves the winner reachable.  The near
// faces are seeds always, the far ones for a non-empty item (fft3.cu:263-293),
// which every item here is.  grid: any, block 256
__global__ void __launch_bounds__(256)
k_bound_ray(const uint4* __restrict__ tbits, int tq, ScoreParams sp, BoundArgs ba, LoopState* ls, DecisionDev* out) {
    pdl_enter();
    BoundState* st = ba.st;
    const BoundEntry en = bound_entry(st);
    if (en.halt || !en.need_ray) return;
    const double head = ba.tab[(size_t)st->win_o * ba.tstride + min((int)(threadIdx.x & 31), 14)];
    const RunHead od = run_head(head);
    const int valid[3] = {(int)__shfl_sync(0xffffffffu, head, 9), (int)__shfl_sync(0xffffffffu, head, 10),
                          (int)__shfl_sync(0xffffffffu, head, 11)};
    const int t = st->win_t;
    const int at[3] = {t / (sp.nz * sp.ny), (t / sp.nz) % sp.ny, t % sp.nz};
    int len[6], total = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        len[k] = k < 3 ? at[k] : valid[k % 3] - 1 - at[k % 3];
        total += len[k];
    }
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (int e = blockIdx.x * wpb + (threadIdx.x >> 5); e < total; e += gridDim.x * wpb) {
        int k = 0, i = e, c[3] = {at[0], at[1], at[2]};
#pragma unroll
        for (int q = 0; q < 5; ++q)
            if (k == q && i >= len[q]) { i -= len[q]; k = q + 1; }
#pragma unroll
        for (int a = 0; a < 3; ++a)
            if (k % 3 == a) c[a] += k < 3 ? -1 - i : 1 + i;
        unsigned int blocked = 0u;   // as one lane sees it: other warps are adding to it
        if (lane == 0) blocked = *(volatile unsigned int*)&st->blocked;
        if (__shfl_sync(0xffffffffu, blocked, 0) >> k & 1u) continue;
        if (!bound_free(od, (const uint32_t*)tbits, 4 * tq, sp.ny, c[0], c[1], c[2]) && lane == 0)
            atomicOr(&st->blocked, 1u << k);
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicInc(&st->rdone, gridDim.x - 1) != gridDim.x - 1) return;
    __threadfence();
    const unsigned int blocked = *(volatile unsigned int*)&st->blocked;
    st->blocked = 0u;
    st->need_ray = 0;
    if ((blocked & 63u) == 63u) {
        st->need_flood = 1;
        return;
    }
    bound_commit(ls, out, sp, st->win_o, t, st->win_s, out->ncand);
}

// Every listed translation checked exactly (one warp each), then, in the last
// CTA to finish, the reference's flood fill (fft3.cu:234-455) over the free
// ones: a breadth-first walk from the seed faces, neighbours along x, y and z
// within the same orientation looked up in a shared-memory hash of the free
// translations.  Blocked and unreached ones get the score 1e300.  The walk
// pushes every translation at most once and a probe visits every slot at most
// once, so both loops are bounded.  More free translations than the table
// takes: the item goes to the union-find flood fill (halt).
// grid: any, block 256, dynamic shared memory bound_flood_smem()
#define PSB_BSLOTS (2 * PSB_BFREE)
inline size_t bound_flood_smem() { return (size_t)PSB_BSLOTS * 8 + (size_t)PSB_BFREE * 4; }
__global__ void __launch_bounds__(256)
k_bound_flood(const uint4* __restrict__ tbits, int tq, ScoreParams sp, BoundArgs ba, int item) {
    pdl_enter();
    BoundState* st = ba.st;
    const BoundEntry en = bound_entry(st);
    if (en.halt || !en.need_flood) return;
    const int count = en.count;
    const int n = count > PSB_BCAP ? 0 : count;   // k_bound_score raises the halt
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5, ny = sp.ny, nz = sp.nz;
    for (int e = blockIdx.x * wpb + (threadIdx.x >> 5); e < n; e += gridDim.x * wpb) {
        const BoundHit h = ba.list[e];
        const int z = h.t % nz, y = (h.t / nz) % ny, x = h.t / (nz * ny);
        if (!bound_free(run_head_of(ba.tab, ba.tstride, h.o), (const uint32_t*)tbits, 4 * tq, ny, x, y, z) && lane == 0)
            ba.list[e].s = 1e300;
    }
    __shared__ int head, tail, nfree, last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicInc(&st->done, gridDim.x - 1) == gridDim.x - 1;
        __threadfence();
        tail = nfree = 0;
    }
    __syncthreads();
    if (!last) return;
    extern __shared__ unsigned int fsm[];
    unsigned int* key = fsm;                  // o * V + t, ~0 empty
    int* val = (int*)(fsm + PSB_BSLOTS);      // list entry, high bit set once reached
    int* queue = val + PSB_BSLOTS;            // slots in walking order
    const unsigned int V = (unsigned int)sp.nx * ny * nz;
    for (int i = threadIdx.x; i < PSB_BSLOTS; i += blockDim.x) key[i] = ~0u;
    __syncthreads();
    auto home = [](unsigned int k) { return (int)((k * 2654435761u) >> 16) & (PSB_BSLOTS - 1); };
    auto find = [&](unsigned int k) {
        int s = home(k);
        for (int i = 0; i < PSB_BSLOTS; ++i, s = (s + 1) & (PSB_BSLOTS - 1)) {
            if (key[s] == k) return s;
            if (key[s] == ~0u) return -1;
        }
        return -1;
    };
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const volatile BoundHit* h = &ba.list[e];
        if (!(h->s < 1e299)) continue;
        if (atomicAdd(&nfree, 1) >= PSB_BFREE) continue;
        const unsigned int k = (unsigned int)h->o * V + (unsigned int)h->t;
        int s = home(k);
        for (int i = 0; i < PSB_BSLOTS; ++i, s = (s + 1) & (PSB_BSLOTS - 1))
            if (atomicCAS(&key[s], ~0u, k) == ~0u) {
                val[s] = e;
                break;
            }
    }
    __syncthreads();
    if (nfree > PSB_BFREE) {
        if (threadIdx.x == 0) {
            st->count = 0;
            st->need_flood = 0;
            st->halt = 1;
            st->halt_item = item;
        }
        return;
    }
    for (int s = threadIdx.x; s < PSB_BSLOTS; s += blockDim.x) {
        if (key[s] == ~0u) continue;
        const double* v = ba.tab + (size_t)(key[s] / V) * ba.tstride + 9;   // numbers of translations
        const int t = (int)(key[s] % V), z = t % nz, y = (t / nz) % ny, x = t / (nz * ny);
        if (x == 0 || y == 0 || z == 0 || x == (int)v[0] - 1 || y == (int)v[1] - 1 || z == (int)v[2] - 1) {
            val[s] |= (int)0x80000000u;
            queue[atomicAdd(&tail, 1)] = s;
        }
    }
    if (threadIdx.x == 0) head = 0;
    __syncthreads();
    while (true) {
        const int h0 = head, h1 = tail;
        __syncthreads();
        if (h0 >= h1) break;
        for (int i = h0 + threadIdx.x; i < h1; i += blockDim.x) {
            const unsigned int k = key[queue[i]];
            const int t = (int)(k % V), z = t % nz, y = (t / nz) % ny, x = t / (nz * ny);
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                // a neighbour outside the tray is no listed translation
                const bool in = d == 0 ? x > 0 : d == 1 ? y > 0 : d == 2 ? z > 0
                              : d == 3 ? x + 1 < sp.nx : d == 4 ? y + 1 < ny : z + 1 < nz;
                if (!in) continue;
                const int step = d % 3 == 0 ? ny * nz : (d % 3 == 1 ? nz : 1);
                const int s = find(d < 3 ? k - step : k + step);
                if (s < 0 || (atomicOr(&val[s], (int)0x80000000u) & (int)0x80000000u)) continue;
                queue[atomicAdd(&tail, 1)] = s;
            }
        }
        if (threadIdx.x == 0) head = h1;
        __syncthreads();
    }
    for (int s = threadIdx.x; s < PSB_BSLOTS; s += blockDim.x)
        if (key[s] != ~0u && val[s] >= 0) ba.list[val[s]].s = 1e300;
}

// The first item of an empty tray: every translation is free and the
// distance field is the far value everywhere, so the score depends on z
// alone, and the first orientation that fits wins at the origin (the smallest
// tie key).  o < 0: none fits.  grid: 1, block 1
__global__ void k_bound_first(int o, double s, ScoreParams sp, LoopState* ls, DecisionDev* out) {
    pdl_enter();
    bound_commit(ls, out, sp, o, 0, s, 0);
}

// The decided placement: each z-run of the item written with its id and
// cleared from the tray's free bits.  Every cell is empty (the translation
// was checked exactly against the same bits).  One warp per run.
// grid: any, block 256
__global__ void __launch_bounds__(256)
k_bound_place(const OrientDesc* __restrict__ orients, const LoopState* __restrict__ ls, int32_t* __restrict__ tray,
              uint32_t* __restrict__ tbits, int tw, int ny, int nz) {
    pdl_enter();
    if (!ls->do_place) return;
    const OrientDesc& od = orients[ls->orient];
    const int px = ls->px, py = ls->py, pz = ls->pz, id = ls->id;
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < od.nruns; r += gridDim.x * wpb) {
        const int4 q = __ldg(&od.runs[r]);
        if (q.w <= 0) continue;
        int a, b, c0, c1;
        orient_run(od, q, &a, &b, &c0, &c1);
        const size_t col = (size_t)(px + a) * ny + (py + b);
        for (int k = pz + c0 + lane; k <= pz + c1; k += 32) tray[col * nz + k] = id;
        const int w = ((pz + c0) >> 5) + lane;
        if (w <= (pz + c1) >> 5) {
            const int z0 = max(pz + c0 - 32 * w, 0), z1 = min(pz + c1 - 32 * w, 31);
            atomicAnd(&tbits[col * tw + w], ~((0xffffffffu << z0) & (0xffffffffu >> (31 - z1))));
        }
    }
}
