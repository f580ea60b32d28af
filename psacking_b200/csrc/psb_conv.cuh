// psb_conv.cuh — the proposal network's layers as register-blocked FP32
// kernels (psb_proposal.cuh holds the network, its inputs, loss and update).
//
// Convolutions: kernel 3, stride 2, padding 1, activations [S][C][D^3], BF16
// weights widened to FP32, FP32 sums.  Written as one FMA chain per thread the
// layers ran at 2-7 TFLOP/s: every FMA fetched its own input from L1, so they
// were load-bound.  Here a CTA keeps its inputs and weights in shared memory
// and a thread a block of results in registers, so that each shared load feeds
// several FMAs: forward 8 positions x 8 channels (64 FMAs per 8 + 2 loads),
// backward-data 2 cells x 8 parities x 4 channels (216 per 12 + 28), and
// backward-weight 4 x 27 weights (108 per 18 + 1).  FP32 throughout.  On the
// tensor cores the FP32 activations would have to be split into three BF16 parts
// (the weights are BF16 already); whether that keeps the present error has not
// been tried.
#pragma once
#include <stdint.h>

#include <type_traits>

#include "psb_pdl.cuh"

// one word to shared memory without waiting for it; zero where ok is false
__device__ __forceinline__ void copy4_async(float* dst, const float* src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(ok ? 4 : 0)
                 : "memory");
}

__device__ __forceinline__ float bf16_up(uint16_t h) { return __uint_as_float((uint32_t)h << 16); }

// The kernels below multiply the zeros around an input, and zero gradients,
// where the layer's definition has no term.  That gives the same sums as long as
// the other factor is finite; a term it is not for makes the sum infinite or NaN.
// So results that are not finite are summed once more, term by term, without
// the terms that do not exist (the functions named _terms, out of line: the
// check is the only cost for ordinary values).
__device__ __forceinline__ bool not_finite(float v) { return !(fabsf(v) < INFINITY); }

// ---------------------------------------------------------------------------
// forward with ReLU
// ---------------------------------------------------------------------------
// one result before the ReLU: sample s, channel co, output position r
template <int CI, int D>
__device__ __noinline__ float conv3_fwd_terms(const float* __restrict__ in, int s, const uint16_t* __restrict__ w,
                                              const float* __restrict__ bias, int co, int r) {
    constexpr int Do = D / 2;
    const int od = r / (Do * Do), oh = r / Do % Do, ow = r % Do;
    float acc = bias[co];
#pragma unroll 1
    for (int ct = 0; ct < CI * 27; ++ct) {
        const int t = ct % 27, id = 2 * od - 1 + t / 9, ih = 2 * oh - 1 + t / 3 % 3, iw = 2 * ow - 1 + t % 3;
        if (id < 0 || ih < 0 || iw < 0) continue;
        acc = fmaf(in[((((size_t)s * CI + ct / 27) * D + id) * D + ih) * D + iw], bf16_up(w[(size_t)co * CI * 27 + ct]), acc);
    }
    return acc;
}

// A CTA computes all CO channels of VPC consecutive output positions (of one
// sample's SL output slabs, or of NS whole samples), CH input channels at a
// time.  The staged input has a zero row at index 0 of each axis (the padding;
// the far side needs none) and each row holds its odd entries behind its even
// ones, so neighbouring output positions read neighbouring words.
// Per result the sum runs over channels, then taps, from the bias on.
// Two CTAs per SM (128 registers): one sums while the other stages.  At 1,536
// samples, layers 1 to 4: 277, 722, 332 and 237 us against 385, 849, 371 and 316
// with one CTA of the first two and weights read down their columns (a sector
// per lane).
template <int CI, int D, int CO, int TV, int CH>
struct ConvFwd {
    static constexpr int Do = D / 2, Do2 = Do * Do, Do3 = Do2 * Do;
    static constexpr int NG = CO / 8, NV = 256 / NG, VPC = NV * TV;
    static constexpr int SL = VPC < Do3 ? VPC / Do2 : Do;       // output slabs per sample part
    static constexpr int NS = VPC < Do3 ? 1 : VPC / Do3;        // samples per CTA
    static constexpr int IS = 2 * SL + 1, P = D + 1, HALF = (P + 1) / 2;   // staged slabs, row length
    static constexpr int ROW = 2 * HALF, SLAB = P * ROW, CHAN = IS * SLAB;
    static constexpr int WR = CO + 4;   // a staged row of weights; padded for the stores, which go down a column
    static constexpr size_t smem = sizeof(float) * ((size_t)NS * CH * CHAN + (size_t)CH * 27 * WR);
    static_assert(VPC % Do2 == 0 && (VPC < Do3 ? Do3 % VPC == 0 : VPC % Do3 == 0) && CI % CH == 0, "tile");
};

template <int CI, int D, int CO, int TV, int CH>
__global__ void __launch_bounds__(256, 2)
k_conv3_fwd(const float* __restrict__ in, int S, const uint16_t* __restrict__ w, const float* __restrict__ bias,
            float* __restrict__ out) {
    pdl_enter();
    using C = ConvFwd<CI, D, CO, TV, CH>;
    extern __shared__ float4 csm4[];
    float* ws = (float*)csm4;                    // [CH][27][WR]
    float* xs = ws + CH * 27 * C::WR;               // [NS][CH][IS][P][ROW]
    const int tid = threadIdx.x, vt = tid % C::NV, g = tid / C::NV;
    const long long v0 = (long long)blockIdx.x * C::VPC;
    const int s0 = (int)(v0 / C::Do3), od0 = (int)(v0 % C::Do3) / C::Do2;
    const int ns = min(C::NS, S - s0);
    float acc[TV][8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const float b = bias[8 * g + c];
#pragma unroll
        for (int i = 0; i < TV; ++i) acc[i][c] = b;
    }
    int at[TV];   // staged offset of each position's window
#pragma unroll
    for (int i = 0; i < TV; ++i) {
        const int r = vt + i * C::NV, s = r / (C::SL * C::Do2), q = r % (C::SL * C::Do2);
        at[i] = s * CH * C::CHAN + 2 * (q / C::Do2) * C::SLAB + 2 * (q / C::Do % C::Do) * C::ROW + q % C::Do;
    }
    for (int i = tid; i < C::NS * CH * C::CHAN; i += 256) xs[i] = 0.f;   // the padding stays zero
    __syncthreads();
    for (int c0 = 0; c0 < CI; c0 += CH) {
#pragma unroll 9
        for (int i = tid; i < CH * 27 * CO; i += 256) {
            const int ct = i % (CH * 27), co = i / (CH * 27);
            ws[ct * C::WR + co] = bf16_up(w[((size_t)co * CI + c0) * 27 + ct]);
        }
        // rows id = 2 od0 - 1 .. of each channel; staged index = id - (2 od0 - 1)
        constexpr int ROWS = C::IS * D;
#pragma unroll 4
        for (int i = tid; i < ns * CH * ROWS * (D / 4); i += 256) {
            const int k4 = i % (D / 4), r = i / (D / 4) % ROWS, sc = i / (D / 4 * ROWS);
            const int sl = r / D, ih = r % D, id = 2 * od0 - 1 + sl;
            if (id < 0 || id >= D) continue;
            const int s = sc / CH, c = sc % CH;
            const float4 v = __ldg((const float4*)(in + (((size_t)(s0 + s) * CI + c0 + c) * D + id) * D * D +
                                                   (size_t)ih * D) + k4);
            float* x = xs + (s * CH + c) * C::CHAN + sl * C::SLAB + (ih + 1) * C::ROW;
            // entry iw sits at padded index iw + 1: odd ones in the second half
            x[C::HALF + 2 * k4] = v.x;
            x[2 * k4 + 1] = v.y;
            x[C::HALF + 2 * k4 + 1] = v.z;
            x[2 * k4 + 2] = v.w;
        }
        __syncthreads();
#pragma unroll 1
        for (int c = 0; c < CH; ++c) {
            const float* xc = xs + c * C::CHAN;
            const float4* wc = (const float4*)(ws + c * 27 * C::WR + 8 * g);
#pragma unroll
            for (int t = 0; t < 27; ++t) {
                const int kd = t / 9, kh = t / 3 % 3, kw = t % 3;
                const int off = kd * C::SLAB + kh * C::ROW + (kw == 1 ? C::HALF : kw / 2);
                const float4 wa = wc[t * (C::WR / 4)], wb = wc[t * (C::WR / 4) + 1];
#pragma unroll
                for (int i = 0; i < TV; ++i) {
                    const float x = xc[at[i] + off];
                    acc[i][0] = fmaf(x, wa.x, acc[i][0]);
                    acc[i][1] = fmaf(x, wa.y, acc[i][1]);
                    acc[i][2] = fmaf(x, wa.z, acc[i][2]);
                    acc[i][3] = fmaf(x, wa.w, acc[i][3]);
                    acc[i][4] = fmaf(x, wb.x, acc[i][4]);
                    acc[i][5] = fmaf(x, wb.y, acc[i][5]);
                    acc[i][6] = fmaf(x, wb.z, acc[i][6]);
                    acc[i][7] = fmaf(x, wb.w, acc[i][7]);
                }
            }
        }
        __syncthreads();
    }
    bool again = false;
#pragma unroll
    for (int i = 0; i < TV; ++i) {
        const int r = vt + i * C::NV, s = r / (C::SL * C::Do2), q = r % (C::SL * C::Do2) + od0 * C::Do2;
        if (s >= ns) continue;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            again = again || not_finite(acc[i][c]);
            out[((size_t)(s0 + s) * CO + 8 * g + c) * C::Do3 + q] = fmaxf(acc[i][c], 0.f);
        }
    }
    if (!again) return;
#pragma unroll 1
    for (int e = 0; e < 8 * TV; ++e) {
        const int r = vt + e / 8 * C::NV, s = r / (C::SL * C::Do2), q = r % (C::SL * C::Do2) + od0 * C::Do2;
        const int co = 8 * g + e % 8;
        if (s < ns)
            out[((size_t)(s0 + s) * CO + co) * C::Do3 + q] = fmaxf(conv3_fwd_terms<CI, D>(in, s0 + s, w, bias, co, q), 0.f);
    }
}

// ---------------------------------------------------------------------------
// gradient w.r.t. the input, times the ReLU mask of that input
// ---------------------------------------------------------------------------
// Input position (2d + pd, ...) collects, per axis, tap 1 of output d when pd
// is 0 and taps 2 of d and 0 of d + 1 when it is 1.  A thread owns two
// neighbouring cells (d, h, w), (d, h, w + 1), all eight parities of each and
// four input channels: 12 output gradients and 27 weights per output channel
// feed 54 FMAs per input channel.  Held to 128 registers for two CTAs per SM
// (with 132 there was one: 1,186 us for 16 <- 32 channels at 1,536 samples,
// 837 with two).  Where the weights of all output channels fit beside the
// gradients (CH = CO) the CTAs stay and take tile after tile, the weights
// staged once: 692 us.
template <int CI, int D, int CO, int CH>
struct ConvBwd {
    static constexpr int Do = D / 2, Do2 = Do * Do, Do3 = Do2 * Do;
    static constexpr int NG = CI / 4, NP = 256 / NG, CELLS = 2 * NP;
    static constexpr int SL = CELLS < Do3 ? CELLS / Do2 : Do;
    static constexpr int NS = CELLS < Do3 ? 1 : CELLS / Do3;
    static constexpr int P = Do + 1, SLAB = P * P, CHAN = (SL + 1) * SLAB;   // zero past the far side
    static constexpr size_t smem = sizeof(float) * ((size_t)NS * CH * CHAN + (size_t)CH * CI * 28);
    static_assert(CELLS % Do2 == 0 && (CELLS < Do3 ? Do3 % CELLS == 0 : CELLS % Do3 == 0) && CO % CH == 0, "tile");
};

// one result before the mask: sample s, channel ci, input position (id, ih, iw)
template <int CI, int D, int CO>
__device__ __noinline__ float conv3_bwd_data_terms(const float* __restrict__ dout, int s, const uint16_t* __restrict__ w,
                                                   int ci, int id, int ih, int iw) {
    constexpr int Do = D / 2, Do3 = Do * Do * Do;
    float acc = 0.f;
#pragma unroll 1
    for (int t = 0; t < 27; ++t) {
        const int ed = id + 1 - t / 9, eh = ih + 1 - t / 3 % 3, ew = iw + 1 - t % 3;   // twice the output position
        if ((ed | eh | ew) & 1 || ed / 2 >= Do || eh / 2 >= Do || ew / 2 >= Do || ed < 0 || eh < 0 || ew < 0) continue;
        const float* g = dout + (size_t)s * CO * Do3 + (ed / 2 * Do + eh / 2) * Do + ew / 2;
#pragma unroll 1
        for (int co = 0; co < CO; ++co) acc = fmaf(g[(size_t)co * Do3], bf16_up(w[((size_t)co * CI + ci) * 27 + t]), acc);
    }
    return acc;
}

template <int CI, int D, int CO, int CH>
__global__ void __launch_bounds__(256, 2)
k_conv3_bwd_data(const float* __restrict__ dout, int S, const uint16_t* __restrict__ w, const float* __restrict__ in,
                 float* __restrict__ din) {
    pdl_enter();
    using C = ConvBwd<CI, D, CO, CH>;
    constexpr int Do = C::Do;
    extern __shared__ float4 csm4[];
    float* ws = (float*)csm4;                    // [CH][CI][28]
    float* gs = ws + CH * CI * 28;               // [NS][CH][SL + 1][P][P]
    const int tid = threadIdx.x, pt = tid % C::NP, g = tid / C::NP;
    const long long ntiles = ((long long)S * C::Do3 + C::CELLS - 1) / C::CELLS;
    // this thread's cell pair
    const int cell = 2 * pt, cs = cell / (C::SL * C::Do2), q = cell % (C::SL * C::Do2);
    const int d = q / C::Do2, h = q / Do % Do, cw = q % Do;
    for (int i = tid; i < C::NS * CH * C::CHAN; i += 256) gs[i] = 0.f;   // the far side stays zero
    __syncthreads();
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long long v0 = tile * C::CELLS;
        const int s0 = (int)(v0 / C::Do3), d0 = (int)(v0 % C::Do3) / C::Do2;
        const int ns = min(C::NS, S - s0);
        float acc[4][2][8];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int p = 0; p < 8; ++p) acc[c][e][p] = 0.f;
        for (int c0 = 0; c0 < CO; c0 += CH) {
            if (CH < CO || tile == blockIdx.x) {
#pragma unroll 4
                for (int i = tid; i < CH * CI * 27; i += 256) {
                    const int t = i % 27, ci = i / 27 % CI, c = i / (27 * CI);
                    ws[(c * CI + ci) * 28 + t] = bf16_up(w[((size_t)(c0 + c) * CI + ci) * 27 + t]);
                }
            }
            constexpr int NVOX = (C::SL + 1) * C::Do2;
#pragma unroll 4
            for (int i = tid; i < ns * CH * NVOX; i += 256) {
                const int r = i % NVOX, sc = i / NVOX, s = sc / CH, c = sc % CH;
                const int od = d0 + r / C::Do2;
                float x = 0.f;
                if (od < Do) x = __ldg(&dout[((size_t)(s0 + s) * CO + c0 + c) * C::Do3 + (size_t)od * C::Do2 + r % C::Do2]);
                gs[(s * CH + c) * C::CHAN + r / C::Do2 * C::SLAB + r / Do % Do * C::P + r % Do] = x;
            }
            __syncthreads();
#pragma unroll 1
            for (int c = 0; c < CH; ++c) {
                const float* gc = gs + (cs * CH + c) * C::CHAN + d * C::SLAB + h * C::P + cw;
                float x[2][2][3];
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int b = 0; b < 2; ++b)
#pragma unroll
                        for (int e = 0; e < 3; ++e) x[a][b][e] = gc[a * C::SLAB + b * C::P + e];
#pragma unroll
                for (int ci = 0; ci < 4; ++ci) {
                    const float4* w4 = (const float4*)(ws + (c * CI + 4 * g + ci) * 28);
                    float wt[28];
#pragma unroll
                    for (int k = 0; k < 7; ++k) {
                        const float4 v = w4[k];
                        wt[4 * k] = v.x;
                        wt[4 * k + 1] = v.y;
                        wt[4 * k + 2] = v.z;
                        wt[4 * k + 3] = v.w;
                    }
#pragma unroll
                    for (int t = 0; t < 27; ++t) {
                        // tap 1: parity 0, output d; tap 2: parity 1, d; tap 0: parity 1, d + 1
                        const int kd = t / 9, kh = t / 3 % 3, kw = t % 3;
                        const int p = (kd != 1) * 4 + (kh != 1) * 2 + (kw != 1);
                        acc[ci][0][p] = fmaf(x[kd == 0][kh == 0][kw == 0], wt[t], acc[ci][0][p]);
                        acc[ci][1][p] = fmaf(x[kd == 0][kh == 0][1 + (kw == 0)], wt[t], acc[ci][1][p]);
                    }
                }
            }
            __syncthreads();
        }
        if (cs >= ns) continue;
        bool again = false;
#pragma unroll
        for (int ci = 0; ci < 4; ++ci) {
            const size_t base = ((size_t)(s0 + cs) * CI + 4 * g + ci) * D * D * D;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
#pragma unroll
                for (int p = 0; p < 4; ++p) again = again || not_finite(acc[ci][p >> 1][2 * r + (p & 1)]);
                const size_t at = base + ((size_t)(2 * (d0 + d) + (r >> 1)) * D + 2 * h + (r & 1)) * D + 2 * cw;
                const float4 m = __ldg((const float4*)(in + at));
                float4 v;
                v.x = !(m.x <= 0.f) ? acc[ci][0][2 * r] : 0.f;
                v.y = !(m.y <= 0.f) ? acc[ci][0][2 * r + 1] : 0.f;
                v.z = !(m.z <= 0.f) ? acc[ci][1][2 * r] : 0.f;
                v.w = !(m.w <= 0.f) ? acc[ci][1][2 * r + 1] : 0.f;
                *(float4*)(din + at) = v;
            }
        }
        if (!again) continue;
#pragma unroll 1
        for (int e = 0; e < 64; ++e) {
            const int ci = 4 * g + e / 16, id = 2 * (d0 + d) + (e >> 3 & 1), ih = 2 * h + (e >> 2 & 1), iw = 2 * cw + (e & 3);
            const size_t at = ((((size_t)(s0 + cs) * CI + ci) * D + id) * D + ih) * D + iw;
            din[at] = in[at] <= 0.f ? 0.f : conv3_bwd_data_terms<CI, D, CO>(dout, s0 + cs, w, ci, id, ih, iw);
        }
    }
}

// ---------------------------------------------------------------------------
// gradient w.r.t. the weights and the bias
// ---------------------------------------------------------------------------
// A thread owns four output channels and all 27 taps of one input channel; the
// CTA's threads cover CG input channels x all CO output channels, NSUB times
// over, each copy taking its share of the staged rows of output positions.
// Along a row the window slides by two inputs, so 18 of its 27 values are new
// per position.  171 registers a thread allow one CTA per SM, so nothing hides a
// load's latency but the CTA itself: the next part's inputs and gradients come by
// asynchronous copies into a second buffer while this part is summed (16 -> 32
// channels at 1,536 samples: 2.28 ms staged in turn with the sums, 0.98 ms so
// with 16 loads in flight, 0.77 ms with two buffers).  grid.x: input channel
// groups, grid.y: shares of the samples; the copies meet in shared memory and
// each CTA adds its sums with one atomic per weight (dw, db zeroed first).
template <int CI, int D, int CO, int CG, int SL, int NS, int SEG>
struct ConvBwdW {
    static constexpr int Do = D / 2, Do2 = Do * Do, Do3 = Do2 * Do;
    static constexpr int NQ = CO / 4, NSUB = 256 / (CG * NQ);
    static constexpr int IS = 2 * SL + 1, P = D + 1, SLAB = P * P, CHAN = IS * SLAB;
    static constexpr int NVOX = SL * Do2, SEGS = NS * NVOX / SEG;
    static constexpr int GR = CO + 4;   // a staged position's gradients: 8 positions x 4 channels on 32 banks
    static constexpr size_t stage = (size_t)NS * NVOX * GR + (size_t)NS * CG * CHAN;
    static constexpr size_t red = (size_t)CG * NQ * 108 + CO;
    static constexpr size_t smem = sizeof(float) * (2 * stage > red ? 2 * stage : red);
    static_assert(256 % (CG * NQ) == 0 && Do % SEG == 0 && Do % SL == 0 && CI % CG == 0, "tile");
    static_assert(NVOX % 8 == 0 && CO % 4 == 0, "staging");
};

// one thread's 27 sums for input channel ci and output channel co over the
// samples [sa, sb); returns the bias sum
template <int CI, int D, int CO>
__device__ __noinline__ float conv3_bwd_weight_terms(const float* __restrict__ dout, const float* __restrict__ in, int sa,
                                                     int sb, int ci, int co, float* __restrict__ sums) {
    constexpr int Do = D / 2, Do3 = Do * Do * Do;
    float b = 0.f;
    for (int t = 0; t < 27; ++t) sums[t] = 0.f;
    for (int s = sa; s < sb; ++s)
        for (int r = 0; r < Do3; ++r) {
            const float g = dout[((size_t)s * CO + co) * Do3 + r];
            if (g == 0.f) continue;
            b += g;
            const int od = r / (Do * Do), oh = r / Do % Do, ow = r % Do;
#pragma unroll 1
            for (int t = 0; t < 27; ++t) {
                const int id = 2 * od - 1 + t / 9, ih = 2 * oh - 1 + t / 3 % 3, iw = 2 * ow - 1 + t % 3;
                if (id < 0 || ih < 0 || iw < 0) continue;
                sums[t] = fmaf(g, in[((((size_t)s * CI + ci) * D + id) * D + ih) * D + iw], sums[t]);
            }
        }
    return b;
}

template <int CI, int D, int CO, int CG, int SL, int NS, int SEG>
__global__ void __launch_bounds__(256)
k_conv3_bwd_weight(const float* __restrict__ dout, const float* __restrict__ in, int S, int chunk,
                   float* __restrict__ dw, float* __restrict__ db) {
    pdl_enter();
    using C = ConvBwdW<CI, D, CO, CG, SL, NS, SEG>;
    constexpr int Do = C::Do;
    extern __shared__ float4 csm4[];
    float* sm = (float*)csm4;                    // 2 x (gs [NS][NVOX][GR], xs [NS][CG][IS][P][P])
    constexpr int GS = NS * C::NVOX * C::GR, XS = NS * CG * C::CHAN;
    const int tid = threadIdx.x, q = tid % C::NQ, cg = tid / C::NQ % CG, sub = tid / (C::NQ * CG);
    const int c0 = blockIdx.x * CG, sa = blockIdx.y * chunk, sb = min(S, sa + chunk);
    const bool bias = blockIdx.x == 0 && cg == 0;
    float acc[4][27], bacc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        bacc[k] = 0.f;
#pragma unroll
        for (int t = 0; t < 27; ++t) acc[k][t] = 0.f;
    }
    for (int i = tid; i < XS; i += 256) sm[2 * GS + i] = sm[2 * GS + XS + i] = 0.f;   // the padding stays zero
    __syncthreads();
    constexpr int PARTS = Do / SL;
    const int steps = sb > sa ? (sb - sa + NS - 1) / NS * PARTS : 0;
    auto stage = [&](int step) {
        const int s0 = sa + step / PARTS * NS, od0 = step % PARTS * SL, ns = min(NS, sb - s0);
        float* gs = sm + step % 2 * GS;
        float* xs = sm + 2 * GS + step % 2 * XS;
        // a warp takes 8 positions x 4 channels: whole sectors, distinct banks
#pragma unroll 4
        for (int i = tid; i < ns * C::NVOX * CO; i += 256) {
            const int v8 = i % 8, c4 = i / 8 % 4, cq = i / 32 % (CO / 4), sv = i / (8 * CO);
            const int c = 4 * cq + c4, s = sv / (C::NVOX / 8), v = sv % (C::NVOX / 8) * 8 + v8;
            copy4_async(gs + (s * C::NVOX + v) * C::GR + c,
                        dout + ((size_t)(s0 + s) * CO + c) * C::Do3 + (size_t)od0 * C::Do2 + v, true);
        }
        constexpr int VIN = C::IS * D * D;
#pragma unroll 4
        for (int i = tid; i < ns * CG * VIN; i += 256) {
            const int v = i % VIN, sc = i / VIN, s = sc / CG, c = sc % CG;
            const int sl = v / (D * D), id = 2 * od0 - 1 + sl;
            const float* src = in + (((size_t)(s0 + s) * CI + c0 + c) * D + max(id, 0)) * D * D + v % (D * D);
            copy4_async(xs + (s * CG + c) * C::CHAN + sl * C::SLAB + (v / D % D + 1) * C::P + v % D + 1, src, id >= 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (steps) stage(0);
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();   // this part has landed for all; the other buffer is read by nobody any more
        if (step + 1 < steps) stage(step + 1);
        const int ns = min(NS, sb - (sa + step / PARTS * NS));
        const float* gs = sm + step % 2 * GS;
        const float* xs = sm + 2 * GS + step % 2 * XS;
        for (int e = sub; e < ns * (C::NVOX / SEG); e += C::NSUB) {
            const int s = e / (C::NVOX / SEG), v = e % (C::NVOX / SEG) * SEG;
            const int sl = v / C::Do2, oh = v / Do % Do, ow = v % Do;
            const float4* gr = (const float4*)(gs + (s * C::NVOX + v) * C::GR) + q;
            const float* x = xs + (s * CG + cg) * C::CHAN + 2 * sl * C::SLAB + 2 * oh * C::P + 2 * ow;
            float win[9][3];
#pragma unroll
            for (int r = 0; r < 9; ++r) win[r][2] = x[r / 3 * C::SLAB + r % 3 * C::P];
#pragma unroll 2
            for (int i = 0; i < SEG; ++i) {
#pragma unroll
                for (int r = 0; r < 9; ++r) {
                    win[r][0] = win[r][2];
                    win[r][1] = x[r / 3 * C::SLAB + r % 3 * C::P + 2 * i + 1];
                    win[r][2] = x[r / 3 * C::SLAB + r % 3 * C::P + 2 * i + 2];
                }
                const float4 g = gr[i * (C::GR / 4)];
                const float gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
#pragma unroll
                    for (int t = 0; t < 27; ++t) acc[k][t] = fmaf(gv[k], win[t / 3][t % 3], acc[k][t]);
                    if (bias) bacc[k] += gv[k];
                }
            }
        }
    }
    bool again = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
#pragma unroll
        for (int t = 0; t < 27; ++t) again = again || not_finite(acc[k][t]);
        again = again || not_finite(bacc[k]);
    }
    again = __syncthreads_or(again);   // the buffers become the sums'
    // the copies' sums, one copy after another
    float* red = sm;                             // [CG * NQ][108], then [CO]
    float* rb = red + CG * C::NQ * 108;
    const int slot = cg * C::NQ + q;
    if (again) {
        for (int p = tid; p < CG * CO; p += 256) {
            const int co = p % CO, ci = p / CO;
            const float b = conv3_bwd_weight_terms<CI, D, CO>(dout, in, sa, sb, c0 + ci, co,
                                                              red + (ci * C::NQ + co / 4) * 108 + co % 4 * 27);
            if (blockIdx.x == 0 && ci == 0) rb[co] = b;
        }
        __syncthreads();
    }
    for (int k = 0; k < (again ? 0 : C::NSUB); ++k) {
        if (sub == k) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
                for (int t = 0; t < 27; ++t) {
                    float* r = red + slot * 108 + j * 27 + t;
                    *r = k == 0 ? acc[j][t] : *r + acc[j][t];
                }
                if (bias) rb[4 * q + j] = k == 0 ? bacc[j] : rb[4 * q + j] + bacc[j];
            }
        }
        __syncthreads();
    }
    for (int i = tid; i < CG * C::NQ * 108; i += 256) {
        const int t = i % 27, j = i / 27 % 4, sq = i / 108, co = 4 * (sq % C::NQ) + j, ci = c0 + sq / C::NQ;
        atomicAdd(&dw[((size_t)co * CI + ci) * 27 + t], red[i]);
    }
    if (blockIdx.x == 0)
        for (int i = tid; i < CO; i += 256) atomicAdd(&db[i], rb[i]);
}

// ---------------------------------------------------------------------------
// linear layers: C[M][N] = sum over k of A(m, k) B(k, n)
// ---------------------------------------------------------------------------
// 16 R x 64 tile per CTA, R x 4 results per thread, BK terms at a time in
// shared memory, the next BK on their way to registers meanwhile.  OP 0: y = x
// W^T + b (A = x [M][K], B = BF16 W [N][K]); OP 1: dx = dy W (A = dy [M][K], B =
// BF16 W [K][N]), times the ReLU mask of x when xmask is given; OP 2: dW = dy^T
// x (A = dy [K][M], B = x [K][N]), grid.z shares of k added with atomics (dW
// zeroed first), with db[m] = sum over k of dy[k][m].
// The layers are a few MFLOP: what bounds them is the chain of K / BK loads, one
// memory latency each where nothing is prefetched, on the few CTAs that N = 64
// leaves.  So the forward layers, whose sum is one chain over K, take R = 1 and
// BK = 32: 512 -> 64 over 1,536 rows 75 -> 27 us, 1,024 -> 64 over 64 rows 144 ->
// 54 us (cold caches).
template <int OP>
struct LinTile {
    static constexpr int R = OP == 0 ? 1 : 4, BK = OP == 0 ? 32 : 16, BM = 16 * R;
};
template <int OP>
__global__ void __launch_bounds__(256)
k_linear(const float* __restrict__ a, const void* __restrict__ b, int M, int N, int K, const float* __restrict__ bias,
         int relu, const float* __restrict__ xmask, float* __restrict__ c, float* __restrict__ db, int kchunk) {
    pdl_enter();
    constexpr int R = LinTile<OP>::R, BK = LinTile<OP>::BK, BM = LinTile<OP>::BM;
    constexpr int NA = BK * BM / 256, NB = BK * 64 / 256;
    __shared__ float As[BK][BM + 4], Bs[BK][68];
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * 64;
    const int ka = OP == 2 ? blockIdx.z * kchunk : 0, kb = OP == 2 ? min(K, ka + kchunk) : K;
    float acc[R][4], bsum = 0.f;
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = OP == 0 && n0 + 4 * tx + j < N ? bias[n0 + 4 * tx + j] : 0.f;
    float pa[NA];
    using TB = std::conditional_t<OP == 2, float, uint16_t>;
    TB pb[NB];   // as loaded: widening here would wait for the load
    // element e of the tiles' loads, along the operand's contiguous index
    auto fetch = [&](int k0) {
#pragma unroll
        for (int e = 0; e < NA; ++e) {
            const int i = tid + 256 * e;
            const int ak = OP == 2 ? i / BM : i % BK, am = OP == 2 ? i % BM : i / BK;
            pa[e] = 0.f;
            if (k0 + ak < kb && m0 + am < M)
                pa[e] = OP == 2 ? a[(size_t)(k0 + ak) * M + m0 + am] : a[(size_t)(m0 + am) * K + k0 + ak];
        }
#pragma unroll
        for (int e = 0; e < NB; ++e) {
            const int i = tid + 256 * e;
            const int bk = OP == 0 ? i % BK : i / 64, bn = OP == 0 ? i / BK : i % 64;
            pb[e] = 0;
            if (k0 + bk < kb && n0 + bn < N)
                pb[e] = ((const TB*)b)[OP == 0 ? (size_t)(n0 + bn) * K + k0 + bk : (size_t)(k0 + bk) * N + n0 + bn];
        }
    };
    fetch(ka);
    for (int k0 = ka; k0 < kb; k0 += BK) {
#pragma unroll
        for (int e = 0; e < NA; ++e) {
            const int i = tid + 256 * e;
            As[OP == 2 ? i / BM : i % BK][OP == 2 ? i % BM : i / BK] = pa[e];
        }
#pragma unroll
        for (int e = 0; e < NB; ++e) {
            const int i = tid + 256 * e;
            float u;
            if constexpr (OP == 2) u = pb[e];
            else u = bf16_up(pb[e]);
            Bs[OP == 0 ? i % BK : i / 64][OP == 0 ? i / BK : i % 64] = u;
        }
        __syncthreads();
        fetch(k0 + BK);   // past kb: zeros, without a load
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            const float4 bv = *(const float4*)&Bs[k][4 * tx];
            const float y[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const float x = As[k][R * ty + i];
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(x, y[j], acc[i][j]);
            }
        }
        if (OP == 2 && blockIdx.x == 0 && tid < BM)
            for (int k = 0; k < BK; ++k) bsum += As[k][tid];
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int m = m0 + R * ty + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + 4 * tx + j;
            if (n >= N) continue;
            const size_t at = (size_t)m * N + n;
            if (OP == 2) atomicAdd(&c[at], acc[i][j]);
            else if (OP == 1) c[at] = xmask && xmask[at] <= 0.f ? 0.f : acc[i][j];
            else c[at] = relu ? fmaxf(acc[i][j], 0.f) : acc[i][j];
        }
    }
    if (OP == 2 && blockIdx.x == 0 && tid < BM && m0 + tid < M) atomicAdd(&db[m0 + tid], bsum);
}
