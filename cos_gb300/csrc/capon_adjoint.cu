// Adjoint of the Capon output power for sm_103a.
//
// With the normalised, loaded covariance R_d = R + d I,
// R = 1/(Ns T) sum_{t,s} x_ts x_ts^H (x_ts the L-sample subarray s of range
// snapshot t), and the MVDR weights w = R_d^-1 a / (a^H R_d^-1 a), the power
// P = 1/(a^H R_d^-1 a) = w^H R_d w is stationary in w, so
//     dP = w^H dR_d w.
// Hence, per pixel, with e_ts = w^H x_ts:
//     dP/d conj(x_t[a]) = 1/(Ns T) sum_s e_ts w_{a-s}        (0 <= a-s < L)
//     dP/dd             = |w|^2
// and, for a per-channel phase x'_m = x_m exp(-j theta_m),
//     dP/dtheta_m       = 2 sum_t Im(conj(dP/dconj(x'_t[m])) x'_t[m]).
// Only the saved weights are needed: the covariance's adjoint is applied in
// factored form through e_ts, so R is neither stored nor rebuilt.
//
// The general kernel's work units are range tiles of one beam (as in the forward
// kernel).  The CTA stages the tile's TILE+2K rows, each warp takes pixels of the tile, and the
// gradient rows are accumulated in shared memory; rows only this tile touches
// are added to the output directly, the 2K rows at each end (shared with the
// neighbouring tiles) with atomics.  Tiles without incoming gradient are
// skipped.
#include "capon_common.cuh"
#include "capon_internal.h"
#include "../../include/cos_capon.h"

namespace cgb {

static constexpr int kAdjWarps = 8;
static constexpr int kAdjTile = 32;

__global__ void __launch_bounds__(32 * kAdjWarps) adjoint_kernel(AdjDev a)
{
    extern __shared__ float2 smem[];
    const int M = a.M, L = a.L, K = a.K, T = 2 * K + 1, Ns = M - L + 1;
    const int rows = kAdjTile + 2 * K;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float2 *xs = smem;                          // rows x M
    float2 *gs = xs + (size_t)rows * M;         // rows x M gradient accumulator
    float *ths = (float *)(gs + (size_t)rows * M);   // M channel sums
    float2 *wbuf = (float2 *)(ths + ((M + 1) & ~1)) + (size_t)warp * (L + T * Ns);
    float2 *ws = wbuf, *es = wbuf + L;
    const float scale = 1.0f / ((float)Ns * (float)T);
    const int tiles_per_beam = (a.Npy + kAdjTile - 1) / kAdjTile;
    const long long units = (long long)a.Nx * tiles_per_beam;
    float dacc = 0.f;

    for (int i = tid; i < M; i += blockDim.x) ths[i] = 0.f;
    for (long long u = blockIdx.x; u < units; u += gridDim.x) {
        const int bx = (int)(u / tiles_per_beam);
        const int p0 = (int)(u % tiles_per_beam) * kAdjTile;
        const int np = min(kAdjTile, a.Npy - p0);
        const int nr = np + 2 * K;
        // skip tiles with no incoming gradient
        bool any = false;
        for (int q = lane; q < np; q += 32) any |= (a.gP[(size_t)bx * a.Npy + p0 + q] != 0.f);
        if (!__syncthreads_or(any)) continue;
        const float2 *xg = a.x + ((size_t)bx * a.Ny + p0) * M;
        for (int i = tid; i < nr * M; i += blockDim.x) {
            xs[i] = xg[i];
            gs[i] = make_float2(0.f, 0.f);
        }
        __syncthreads();
        for (int q = warp; q < np; q += kAdjWarps) {
            const long long pix = (long long)bx * a.Npy + p0 + q;
            const float g = a.gP[pix];
            if (g == 0.f) continue;  // warp-uniform
            float wn = 0.f;
            for (int l = lane; l < L; l += 32) {
                const float2 wl = a.w[(size_t)pix * L + l];
                ws[l] = wl;
                wn += cabs2(wl);
            }
            for (int o = 16; o; o >>= 1) wn += __shfl_xor_sync(0xffffffffu, wn, o);
            if (lane == 0) dacc += g * wn;
            __syncwarp();
            // e_ts = w^H x_ts for the pixel's rows q .. q+2K
            for (int r = lane; r < T * Ns; r += 32) {
                const int t = r / Ns, s = r % Ns;
                const float2 *xt = xs + (size_t)(q + t) * M + s;
                float2 e = make_float2(0.f, 0.f);
                for (int l = 0; l < L; ++l) e = cadd(e, cconjmul(ws[l], xt[l]));
                es[r] = e;
            }
            __syncwarp();
            // dP/dconj(x_t[c]) into the shared accumulator (rows q+t are shared
            // by up to 2K+1 pixels of this tile: shared-memory atomics)
            for (int c = lane; c < M; c += 32) {
                const int s0 = max(0, c - L + 1), s1 = min(Ns - 1, c);
                for (int t = 0; t < T; ++t) {
                    float2 G = make_float2(0.f, 0.f);
                    for (int s = s0; s <= s1; ++s) G = cadd(G, cmul(es[t * Ns + s], ws[c - s]));
                    G = cscale(G, g * scale);
                    float2 *dst = gs + (size_t)(q + t) * M + c;
                    atomicAdd(&dst->x, G.x);
                    atomicAdd(&dst->y, G.y);
                }
            }
            __syncwarp();
        }
        __syncthreads();
        // write the tile's gradient rows; the channel-phase sums use them
        float2 *gout = a.gx + ((size_t)bx * a.Ny + p0) * M;
        for (int i = tid; i < nr * M; i += blockDim.x) {
            const int r = i / M, c = i % M;
            const float2 G = gs[i];
            if (G.x == 0.f && G.y == 0.f) continue;
            const float2 xv = xs[i];
            atomicAdd(&ths[c], 2.f * (G.x * xv.y - G.y * xv.x));
            // rows 0..2K-1 and the last 2K are shared with the neighbouring tiles
            if (r < 2 * K || r >= np) {
                atomicAdd(&gout[i].x, G.x);
                atomicAdd(&gout[i].y, G.y);
            } else {
                const float2 o = gout[i];
                gout[i] = make_float2(o.x + G.x, o.y + G.y);
            }
        }
        __syncthreads();
    }
    if (a.gth)
        for (int i = tid; i < M; i += blockDim.x)
            if (ths[i] != 0.f) atomicAdd(&a.gth[i], ths[i]);
    if (a.gd && lane == 0 && dacc != 0.f) atomicAdd(a.gd, dacc);
}

// The same adjoint by range rows, for L = 8, 16, 24, 32.  A pair (pixel p, window
// row t) adds to row y = p + t only, so a warp owns a row and gathers from the T
// pixels whose window holds it: every pair is formed once, a gradient row is
// complete in its warp, and neither the tile's rows nor the 2K rows between tiles
// need atomics (the tile form above adds every pair into shared memory with
// them).
//
// A lane takes (t, SB consecutive subarrays s) and holds the pixel's L weights in
// registers for both products:
//   e_s = w^H x[s .. s+L-1]      each sample meets w_l for every (s, l) with
//                                s - s0 + l = i: two packed fmas, real and
//                                imaginary part each as a sum over the pair
//                                (w.re, w.im);
//   G[c] += sum_s e_s w_{c-s}    with the same e_s still in registers, over the
//                                SB + L - 1 channels they reach, added to the
//                                row's accumulator of window row t in shared
//                                memory.  At one step the lanes of a t write
//                                different channels, and a warp barrier orders
//                                the steps.  (Gathered by channel, half the
//                                products are with s outside 0 .. Ns-1.)
// The next row's samples and weights arrive by cp.async under this row's products
// (398 -> 335 us together with the gradient rows leaving as vector reductions
// instead of a load and a store).  What bounds it: the FP32 pipe over the useful
// lanes (30 of 32 at M=64, L=32, K=2), issue 58 %.  Gradients at [128][1024][64],
// L=32, K=2: 333 us, 625 us as tiles.
static constexpr int kRowWarps = 8;

struct AdjRowSmem {
    int xs, ws, as;        // strides: samples, weights, accumulators
    size_t off_w, off_a, per_warp, total;
    __host__ __device__ AdjRowSmem(int M, int L, int T, int SB)
    {
        // strides that keep the 16-byte accesses of eight lanes on different
        // banks: of the T pixels' weights, and of the accumulators at SB = 6
        xs = (M + SB + 3) & ~1;      // zero tail: the last block's samples past the row
        ws = L + 2;
        as = ((M + SB - 4 + 15) & ~15) + 4;
        // samples and weights twice: the next row's arrive during this row's products
        off_w = (size_t)2 * xs * sizeof(float2);
        off_a = off_w + (size_t)2 * (T + 1) * ws * sizeof(float2);   // T + 1: lanes without an item
        per_warp = (off_a + (size_t)(T + 1) * as * sizeof(float2) + 15) & ~(size_t)15;
        total = kRowWarps * per_warp + (size_t)kRowWarps * M * sizeof(float);
    }
};

// 8 bytes global to shared, zeros when !is
COS_DEV void async_copy8(void *dst, const void *src, bool is)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(is ? 8 : 0)
                 : "memory");
}

// `per` window rows at a time (at most 32, a lane each): a longer window, or one whose
// accumulators leave fewer than two CTAs an SM, takes several passes over the rows, whose
// gradients add up (backward pass at M=128, L=32, K=4, [64][520]: 840 -> 640 us; M=33, L=16,
// K=17: 444 -> 354 us, both against register-blocked tiles); SINGLE: one is enough, which
// keeps the passes' bounds out of the rows' loop (333 us, 342 without it, in the case
// above).  A row none of whose pixels has a gradient is not staged: the gradients are
// read two rows ahead.
template <int L, int SB, bool SINGLE>
__global__ void __launch_bounds__(32 * kRowWarps, 2) adjoint_row_kernel(AdjDev a, int per)
{
    static_assert(SB % 2 == 0 && L % 2 == 0, "channel pairs are 16 bytes");
    extern __shared__ __align__(16) unsigned char smraw[];
    const int M = a.M, Ns = M - L + 1;
    const AdjRowSmem S(M, L, per, SB);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char *const mine = smraw + warp * S.per_warp;
    float2 *const acc = (float2 *)(mine + S.off_a);
    float *const ths = (float *)(smraw + kRowWarps * S.per_warp) + (size_t)warp * M;   // channel-phase sums
    const float scale = 1.0f / ((float)Ns * (float)(2 * a.K + 1));
    const int nsb = (Ns + SB - 1) / SB;
    // a warp's sum of g |w|^2.  Its terms cancel (gradients of either sign), so they are
    // added in FP64, one a row, and a CTA's sum goes out once
    __shared__ double dsum[kRowWarps];
    double dacc = 0.0;
    for (int c = lane; c < M; c += 32) ths[c] = 0.f;
    for (int b = 0; b < 2; ++b) {   // the zero tails: samples past M, weights of the lanes without an item
        for (int c = M + lane; c < S.xs; c += 32) ((float2 *)mine)[b * S.xs + c] = make_float2(0.f, 0.f);
        for (int l = lane; l < L; l += 32)
            ((float2 *)(mine + S.off_w))[(b * (per + 1) + per) * S.ws + l] = make_float2(0.f, 0.f);
    }
    const unsigned rows = (unsigned)a.Nx * a.Ny, step = gridDim.x * kRowWarps;
#pragma unroll 1
    for (int t0 = 0; t0 < (SINGLE ? 1 : 2 * a.K + 1); t0 += per) {
        const int T = SINGLE ? per : min(per, 2 * a.K + 1 - t0), items = T * nsb;   // window rows t0 .. t0+T-1
        // gradient of pixel y-t0-t on lane t; 0 where there is none
        auto grad = [&](unsigned row) {
            const unsigned bx = row / (unsigned)a.Ny;
            const int p = (int)(row - bx * a.Ny) - t0 - lane;
            return row < rows && lane < T && p >= 0 && p < a.Npy ? a.gP[(size_t)bx * a.Npy + p] : 0.f;
        };
        // the row's samples and the weights of its pixels (zeros where there is none)
        // into buffer b
        auto stage = [&](unsigned row, int b) {
            const unsigned bx = row / (unsigned)a.Ny;
            const int y = (int)(row - bx * a.Ny);
            float2 *const xd = (float2 *)mine + b * S.xs, *const wd = (float2 *)(mine + S.off_w) + b * (per + 1) * S.ws;
            const float2 *xr = a.x + (size_t)row * M;
            for (int c = lane; c < M; c += 32) async_copy8(xd + c, xr + c, true);
            for (int i = lane; i < T * L; i += 32) {
                const int t = i / L, l = i % L, p = y - t0 - t;
                const bool is = p >= 0 && p < a.Npy;
                async_copy8(wd + t * S.ws + l, a.w + ((size_t)bx * a.Npy + (is ? p : 0)) * L + l, is);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        unsigned row = blockIdx.x * kRowWarps + warp;
        float gnext = grad(row), gafter = grad(row + step);
        unsigned next = __ballot_sync(0xffffffffu, gnext != 0.f);
        __syncwarp();   // the last pass' readers are done
        if (next) stage(row, 0);
        int b = 0;
        for (; row < rows; row += step, b ^= 1) {
            const float gl = gnext;
            gnext = gafter;
            gafter = grad(row + 2 * step);
            // a pixel without a gradient takes no part, its weights finite or not; a row
            // of such pixels gets nothing
            const unsigned on = next;
            next = __ballot_sync(0xffffffffu, gnext != 0.f);
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncwarp();   // the row has arrived for every lane, and the last one's readers are done
            if (next) stage(row + step, b ^ 1);
            if (on == 0u) continue;
            const float2 *const xw = (const float2 *)mine + b * S.xs;
            float2 *const ws = (float2 *)(mine + S.off_w) + b * (per + 1) * S.ws;
            for (int t = 0; t < T; ++t)
                if (!(on >> t & 1u))
                    for (int l = lane; l < L; l += 32) ws[t * S.ws + l] = make_float2(0.f, 0.f);
            for (int i = lane; i < (T + 1) * S.as; i += 32) acc[i] = make_float2(0.f, 0.f);
            __syncwarp();
            for (int it0 = 0; it0 < items; it0 += 32) {
                const int it = it0 + lane, t = it < items ? it / nsb : per, s0 = it < items ? (it - t * nsb) * SB : 0;
                const float gt = __shfl_sync(0xffffffffu, gl, t < T ? t : 0), g = t < T ? gt : 0.f;
                float2 w[L];
#pragma unroll
                for (int l = 0; l < L; l += 2) {
                    const float4 v = *(const float4 *)(ws + t * S.ws + l);
                    w[l] = make_float2(v.x, v.y);
                    w[l + 1] = make_float2(v.z, v.w);
                }
                if (t0 == 0 && it < nsb) {   // pixel y; one lane adds g |w|^2
                    float wn = 0.f;
#pragma unroll
                    for (int l = 0; l < L; ++l) wn += cabs2(w[l]);
                    if (it == 0) dacc += (double)(g * wn);
                }
                // e_s, s = s0 .. s0+SB-1: (re, im) parts as pair sums
                float2 er[SB], ei[SB];
#pragma unroll
                for (int j = 0; j < SB; ++j) er[j] = ei[j] = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < SB + L - 1; i += 2) {
                    const float4 q = *(const float4 *)(xw + s0 + i);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float2 v = h ? make_float2(q.z, q.w) : make_float2(q.x, q.y);
                        const float2 u = make_float2(v.y, -v.x);
#pragma unroll
                        for (int j = 0; j < SB; ++j) {
                            const int l = i + h - j;
                            if (l >= 0 && l < L) {
                                // conj(w) v = (w.re v.re + w.im v.im, w.re v.im - w.im v.re)
                                er[j] = ffma2(w[l], v, er[j]);
                                ei[j] = ffma2(w[l], u, ei[j]);
                            }
                        }
                    }
                }
                // e_s g / (Ns T) as (re, -im) and (im, re)
                const float gs = g * scale;
#pragma unroll
                for (int j = 0; j < SB; ++j) {
                    const bool in = s0 + j < Ns;
                    const float re = in ? (er[j].x + er[j].y) * gs : 0.f, im = in ? (ei[j].x + ei[j].y) * gs : 0.f;
                    er[j] = make_float2(re, -im);
                    ei[j] = make_float2(im, re);
                }
                float2 *const at = acc + (SINGLE ? t : min(t, T)) * S.as + s0;   // lanes without an item: past the last
#pragma unroll
                for (int i = 0; i < SB + L - 1; i += 2) {
                    float2 G[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float2 pr = make_float2(0.f, 0.f), pi = pr;
#pragma unroll
                        for (int j = 0; j < SB; ++j) {
                            const int l = i + h - j;
                            if (l >= 0 && l < L) {
                                pr = ffma2(er[j], w[l], pr);
                                pi = ffma2(ei[j], w[l], pi);
                            }
                        }
                        G[h] = make_float2(pr.x + pr.y, pi.x + pi.y);
                    }
                    float4 *const d = (float4 *)(at + i);
                    const float4 o = *d;
                    *d = make_float4(o.x + G[0].x, o.y + G[0].y, o.z + G[1].x, o.w + G[1].y);
                    __syncwarp();
                }
            }
            // the row's gradient, and its share of the channel phases
            float2 *gout = a.gx + (size_t)row * M;
            for (int c = lane; c < M; c += 32) {
                float2 G = acc[c];
                for (int t = 1; t < T; ++t) G = cadd(G, acc[t * S.as + c]);
                const float2 xv = xw[c];
                ths[c] += 2.f * (G.x * xv.y - G.y * xv.x);
                // added without waiting for the old value
                asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(gout + c), "f"(G.x), "f"(G.y) : "memory");
            }
        }
    }
    if (lane == 0) dsum[warp] = dacc;
    __syncthreads();
    if (a.gd && threadIdx.x == 0) {
        double v = 0.0;
        for (int k = 0; k < kRowWarps; ++k) v += dsum[k];
        if (v != 0.0) atomicAdd(a.gd, (float)v);
    }
    if (a.gth) {
        const float *all = (const float *)(smraw + kRowWarps * S.per_warp);
        for (int c = threadIdx.x; c < M; c += blockDim.x) {
            float v = 0.f;
            for (int k = 0; k < kRowWarps; ++k) v += all[(size_t)k * M + c];
            if (v != 0.f) atomicAdd(&a.gth[c], v);
        }
    }
}

template <class Kern, class... Args>
static int launch_adjoint_with(Kern kern, const AdjDev &a, long long units, size_t smem, int num_sms, cudaStream_t s,
                               Args... args)
{
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kAdjWarps, smem);
    if (e != cudaSuccess) return e;
    long long grid = (long long)num_sms * (per_sm > 0 ? per_sm : 1);
    if (grid > units) grid = units;
    kern<<<(unsigned)grid, 32 * kAdjWarps, smem, s>>>(a, args...);
    return cudaGetLastError();
}

// window rows a pass of the row kernel takes: at most 32 (a lane each) and what
// leaves two CTAs an SM, spread evenly over the passes.  0: not even one row fits so
static int rows_per_pass(const AdjDev &a)
{
    const int T = 2 * a.K + 1;
    int most = T < 32 ? T : 32;
    while (most > 0 && AdjRowSmem(a.M, a.L, most, 8).total > 112 * 1024) --most;
    if (most == 0) return 0;
    const int passes = (T + most - 1) / most;
    return (T + passes - 1) / passes;
}

// SB: the block length that keeps the lanes fullest, passes of 32 items by the
// products of an item
template <int L>
static int launch_rows(const AdjDev &a, int per, int num_sms, cudaStream_t s)
{
    static_assert(kRowWarps == kAdjWarps, "one launch helper");
    const int Ns = a.M - L + 1;
    const long long units = ((long long)a.Nx * a.Ny + kRowWarps - 1) / kRowWarps;
    auto cost = [&](int sb) { return (per * ((Ns + sb - 1) / sb) + 31) / 32 * (sb + 2); };
    int best = 2;
    for (int sb : {4, 6, 8})
        if (cost(sb) < cost(best)) best = sb;
    const size_t smem = AdjRowSmem(a.M, L, per, best).total;
    auto go = [&](auto kern) { return launch_adjoint_with(kern, a, units, smem, num_sms, s, per); };
    const bool single = per == 2 * a.K + 1;
    return best == 2   ? single ? go(adjoint_row_kernel<L, 2, true>) : go(adjoint_row_kernel<L, 2, false>)
           : best == 4 ? single ? go(adjoint_row_kernel<L, 4, true>) : go(adjoint_row_kernel<L, 4, false>)
           : best == 6 ? single ? go(adjoint_row_kernel<L, 6, true>) : go(adjoint_row_kernel<L, 6, false>)
                       : single ? go(adjoint_row_kernel<L, 8, true>) : go(adjoint_row_kernel<L, 8, false>);
}

int launch_adjoint(const AdjDev &a, int num_sms, cudaStream_t s)
{
    const int T = 2 * a.K + 1, Ns = a.M - a.L + 1, rows = kAdjTile + 2 * a.K;
    const size_t smem = (size_t)2 * rows * a.M * sizeof(float2) + (size_t)((a.M + 1) & ~1) * sizeof(float) +
                        (size_t)kAdjWarps * (a.L + T * Ns) * sizeof(float2);
    if (smem > 227 * 1024 || a.L > 64) return cudaErrorNotSupported;
    // by rows (counted in 32 bits, two steps of the grid ahead); the tiles serve the other
    // subarray lengths
    const int per = (long long)a.Nx * a.Ny < 0xffffffffLL - (1 << 20) ? rows_per_pass(a) : 0;
    if (per) {
        switch (a.L) {
        case 8: return launch_rows<8>(a, per, num_sms, s);
        case 16: return launch_rows<16>(a, per, num_sms, s);
        case 24: return launch_rows<24>(a, per, num_sms, s);
        case 32: return launch_rows<32>(a, per, num_sms, s);
        default: break;
        }
    }
    const long long units = (long long)a.Nx * ((a.Npy + kAdjTile - 1) / kAdjTile);
    return launch_adjoint_with(adjoint_kernel, a, units, smem, num_sms, s);
}

}  // namespace cgb
