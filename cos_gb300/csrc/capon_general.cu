// General element-space path for sm_103a: z, P and w for the frames without a
// fused instantiation -- any subarray length L <= 64, any window, and
// forward-backward averaging.
//
//   1. covariance kernel (this file): R per pixel, float-float sums of exact
//      products, rounded once, to HBM/L2 as the solve stage's records;
//   2. solve kernel (capon_general.cuh): FP32 Cholesky in registers and the
//      outputs.
//
// Covariance.  Along diagonal d of one range row y,
//   r_y[k,k+d] = sum_{i=k}^{k+Ns-1} x_y[i] conj(x_y[i+d]),   R = sum_{y<T} r_{p+y},
// (the smoothing and temporal averaging of getCaponC.pyx:197-242).  The precise
// pipeline, which this one replaces where no refinement is wanted, slides along
// the diagonals of every pixel's whole window; here a row's sums are formed once for
// all the pixels whose window holds the row:
//   rows     a thread owns a diagonal of a row, r[0] from Ns products, then
//            r[k] = r[k-1] + x[k-1+Ns] conj(..) - x[k-1] conj(..), all in
//            float-float with the products exact (ff_cmacc); (value, remainder) to
//            shared memory.  Products are formed anew for each slide: stored
//            between the two, they would need more room than the sums;
//   windows  a thread owns an entry and walks the tile's pixels with the last T
//            row sums in registers, adds them in float-float and rounds once.
//            Forward-backward averaging, (R + J R^T J)/2, pairs entry k with
//            entry L-1-d-k of the same diagonal: a thread sums both and writes
//            the mean to both.
// Only R itself is rounded, as in the precise pipeline.  (FP32 window sums of T
// products, float-float from there, are a tenth faster, but their errors are the
// same all along a diagonal and add up in P: 1.2 to 1.45 times as far from 64 bits for
// K = 2 to 12, R itself 1.1 to 3.5 times.)
// What bounds it: the FMA pipe, about 57 k packed operations a pixel at M=64, L=32,
// K=2 with forward-backward averaging, at 50 to 65 % of its rate (issue 49 %, L1 59 %),
// with waits at the barriers between the phases; what fits of the row sums into shared
// memory gives the threads of a phase.  Measured, 60 k pixels at M=48, L=24, K=2 with
// weights: 1.44 ms in the precise pipeline, 0.21 ms here + 0.15 ms in the solve stage; 65 k
// pixels at M=64, L=32, K=2 with forward-backward averaging: 2.56 ms, 0.38 + 0.20 ms.
#include <algorithm>
#include <cmath>

#include "capon_common.cuh"
#include "capon_general.cuh"
#include "capon_internal.h"
#include "../../include/cos_capon.h"

namespace cgb {

using GeneralSolve = int(const FrameDev &, const float2 *, unsigned *, int, cudaStream_t);
GeneralSolve general_solve_l8_zp, general_solve_l8_w, general_solve_l16_zp, general_solve_l16_w, general_solve_l24_zp,
    general_solve_l24_w, general_solve_l32_zp, general_solve_l32_w, general_solve_l48_zp, general_solve_l48_w,
    general_solve_l64_zp, general_solve_l64_w;

namespace {

using general::Record;

constexpr int kCovThreads = 256;
constexpr int kCovParts = 16;   // the most chunks of a unit's diagonals

// A pair of diagonals p and L-1-p has L + 1 entries, whatever p is, and shares the
// storage of a row: entry (k, p) is entry k of pair p, entry (k, L-1-p) entry L - k.
struct CovShape {
    int tile, rows;    // pixels per unit and their range rows
    int pairs;         // pairs in shared memory at a time
    int seg, nseg;     // pixels per item of the window sums, items along the tile
    // strides: samples of a row, entries of a pair, of a row's pairs; odd, so that the
    // lanes of a load or store, on neighbouring rows or diagonals, fall on different banks
    int XS, PE, RS;
    size_t off_r, off_tab, off_tr, total;
    __host__ __device__ CovShape(int tile_, int pairs_, int K, int M, int L)
    {
        tile = tile_;
        rows = tile + 2 * K;
        pairs = pairs_;
        seg = tile;
        nseg = 1;
        XS = (M + 1) | 1;
        PE = (L + 1) | 1;
        RS = (pairs * PE) | 1;
        off_r = ((size_t)rows * XS * sizeof(float2) + 15) & ~(size_t)15;
        off_tab = off_r + (size_t)rows * RS * sizeof(float4);
        off_tr = off_tab + (((size_t)pairs * (L + 1) * sizeof(unsigned short) + 15) & ~(size_t)15);
        total = off_tr + (size_t)rows * sizeof(float2);
    }
};

// (h, l) += a b, componentwise, the product exact: TwoSum with the rounded product,
// whose own error comes with its last difference, a b - bb, in one fma
COS_DEV void ff_fma2(float2 &h, float2 &l, float2 a, float2 b)
{
    const float2 s = fadd2(h, ffma2(a, b, make_float2(0.f, 0.f))), n = fsub2(h, s), t = fadd2(s, n);
    l = fadd2(l, fadd2(fsub2(h, t), ffma2(a, b, n)));
    h = s;
}
// (h, l) += x conj(y)
COS_DEV void ff_cmacc(float2 &h, float2 &l, float2 x, float2 y)
{
    ff_fma2(h, l, x, make_float2(y.x, y.x));
    ff_fma2(h, l, make_float2(x.y, -x.x), make_float2(y.y, y.y));
}
COS_DEV void ff_add(float2 &h, float2 &l, float4 v)
{
    two_sum_acc(h, l, make_float2(v.x, v.y));
    l = fadd2(l, make_float2(v.z, v.w));
}

// T: the temporal window 2K+1, 0 = taken from the frame (the row ring of the window
// sums needs a compile-time length; without it a pixel reads all its rows)
template <int T_, bool FB>
__global__ void __launch_bounds__(kCovThreads, 2)
cov_kernel(FrameDev f, CovShape S, float2 *__restrict__ work, int units)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const int M = f.M, L = f.L, K = T_ ? (T_ - 1) / 2 : f.K, T = 2 * K + 1, Ns = M - L + 1;
    const int XS = S.XS, PE = S.PE, RS = S.RS, tid = threadIdx.x, rec = Record::size(L);
    const int half = (L + 1) / 2;
    float2 *xs = (float2 *)smraw;
    float4 *Rr = (float4 *)(smraw + S.off_r);                     // [row][pair][entry] (value, remainder)
    unsigned short *tab = (unsigned short *)(smraw + S.off_tab);  // the chunk's entries k << 8 | d
    float2 *tr = (float2 *)(smraw + S.off_tr);                    // tr(R) of a row, value and remainder
    __shared__ int s_count;
    const int tiles_per_beam = (f.Npy + S.tile - 1) / S.tile;
    const float inv_L = 1.f / (float)L, inv_M = 1.f / (float)M;
    // the entries of pairs p0 .. p0+np-1 in the record's order, for the window sums;
    // with forward-backward averaging the first of each mirrored two
    auto table = [&](int p0, int np) {
        const int a0 = p0, a1 = p0 + np, b0 = max(L - p0 - np, a1), b1 = L - p0;   // diagonals [a0, a1), [b0, b1)
        // of row k: d < L - k, or, as 2k <= L-1-d says, d < L - 2k
        auto most = [&](int k) { return FB ? L - 2 * k : L - k; };
        auto count = [&](int k) { return max(0, min(a1, most(k)) - a0) + max(0, min(b1, most(k)) - b0); };
        for (int k = tid; k < L; k += kCovThreads) {
            int off = 0;
            for (int i = 0; i < k; ++i) off += count(i);
            for (int d = a0; d < min(a1, most(k)); ++d) tab[off++] = (unsigned short)(k << 8 | d);
            for (int d = b0; d < min(b1, most(k)); ++d) tab[off++] = (unsigned short)(k << 8 | d);
            if (k == L - 1) s_count = off;
        }
    };
    if (S.pairs >= half) table(0, half);
#pragma unroll 1
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
        const int bx = u / tiles_per_beam, q0 = (u % tiles_per_beam) * S.tile;
        const int np = min(S.tile, f.Npy - q0), rows = np + 2 * K;
        const size_t pix0 = (size_t)bx * f.Npy + q0;
        const float2 *src = f.x + ((size_t)bx * f.Ny + q0) * M;
        for (int i = tid; i < rows * M; i += kCovThreads) {
            const int r = small_div(i, inv_M);
            xs[r * XS + (i - r * M)] = src[i];
        }
#pragma unroll 1
        for (int p0 = 0; p0 < half; p0 += S.pairs) {
            const int pairs = min(S.pairs, half - p0);
            const float inv_pairs = 1.f / (float)pairs;
            if (S.pairs < half) table(p0, pairs);
            __syncthreads();
            // ---- rows: the smoothing sums of one diagonal of one range row, the chunk's
            // long diagonals first
            const float inv_rows = 1.f / (float)rows;
#pragma unroll 1
            for (int it = tid; it < 2 * pairs * rows; it += kCovThreads) {
                const int j = small_div(it, inv_rows), r = it - j * rows;
                const bool second = j >= pairs;
                const int p = p0 + (second ? j - pairs : j), d = second ? L - 1 - p : p;
                if (second && 2 * p == L - 1) continue;   // the middle diagonal of an odd L, alone
                const float2 *const xi = xs + r * XS, *const xj = xi + d;
                float4 *o = Rr + (size_t)r * RS + (p - p0) * PE + (second ? L : 0);
                const int step = second ? -1 : 1;
                float2 h = make_float2(0.f, 0.f), l = h;
#pragma unroll 4
                for (int i = 0; i < Ns; ++i) ff_cmacc(h, l, xi[i], xj[i]);
                *o = make_float4(h.x, h.y, l.x, l.y);
                // the next step's samples are loaded under this one's sums (the last
                // load, one past the row, is not used)
                float2 ax = xi[Ns], ay = xj[Ns], sx = xi[0], sy = xj[0];
#pragma unroll 1
                for (int k = 1; k < L - d; ++k) {
                    const float2 nax = xi[k + Ns], nay = xj[k + Ns], nsx = xi[k], nsy = xj[k];
                    ff_cmacc(h, l, ax, ay);
                    ff_cmacc(h, l, sx, make_float2(-sy.x, -sy.y));
                    o += step;
                    *o = make_float4(h.x, h.y, l.x, l.y);
                    ax = nax;
                    ay = nay;
                    sx = nsx;
                    sy = nsy;
                }
            }
            // subarray means of the centre rows, g[l] = (1/Ns) sum_s x[s+l]
            // (getCaponC.pyx:246-255)
            if (p0 == 0) {
                const float invNs = 1.f / (float)Ns;
#pragma unroll 1
                for (int it = tid; it < np * L; it += kCovThreads) {
                    const int p = small_div(it, inv_L), l = it - p * L;
                    const float2 *xr = xs + (p + K) * XS + l;
                    float2 g0 = make_float2(0.f, 0.f), g1 = g0;
                    int s = 0;
                    for (; s + 1 < Ns; s += 2) {
                        g0 = fadd2(g0, xr[s]);
                        g1 = fadd2(g1, xr[s + 1]);
                    }
                    if (s < Ns) g0 = fadd2(g0, xr[s]);
                    work[(pix0 + p) * rec + Record::mean(L) + l] = cscale(fadd2(g0, g1), invNs);
                }
            }
            __syncthreads();
            // ---- tr(R) of a row, a warp each: diagonal 0 is the first half of pair 0
            if (p0 == 0) {
                for (int r = tid >> 5; r < rows; r += kCovThreads / 32) {
                    float2 v = make_float2(0.f, 0.f);   // (value, remainder)
                    auto add = [&](float a, float e) {
                        const float s = v.x + a, b = s - v.x;
                        v = make_float2(s, v.y + ((v.x - (s - b)) + (a - b)) + e);
                    };
                    for (int k = tid & 31; k < L; k += 32) {
                        const float4 e = Rr[(size_t)r * RS + k];
                        add(e.x, e.z);
                    }
                    for (int w = 16; w; w >>= 1) {
                        const float2 t = shfl2_xor(v, w, 32);
                        add(t.x, t.y);
                    }
                    if ((tid & 31) == 0) tr[r] = v;
                }
            }
            // ---- window sums of the tile's pixels, rounded once
            const int entries = s_count;
            const float inv_entries = 1.f / (float)entries;
#pragma unroll 1
            for (int it = tid; it < entries * S.nseg; it += kCovThreads) {
                const int sg = small_div(it, inv_entries), e = tab[it - sg * entries];
                const int k = e >> 8, d = e & 255, km = L - 1 - d - k;   // km: the mirror of k on its diagonal
                const int s0 = sg * S.seg, sp = min(S.seg, np - s0);
                const float4 *const rd = Rr + (size_t)s0 * RS + (d < half ? (d - p0) * PE : (L - 1 - d - p0) * PE + L);
                const float4 *ra = d < half ? rd + k : rd - k, *rb = d < half ? rd + km : rd - km;
                float2 *out = work + (pix0 + s0) * rec + Record::row(k, L) + d;
                const int mirror = Record::row(km, L) - Record::row(k, L);
                auto put = [&](float2 h, float2 l) __attribute__((always_inline)) {
                    float2 v = fadd2(h, l);
                    if (FB) {
                        v = cscale(v, 0.5f);
                        out[mirror] = v;
                    }
                    *out = v;
                    out += rec;
                };
                if constexpr (T_ != 0) {
                    float4 ring[T_], mir[FB ? T_ : 1];
                    const int nr = sp + T_ - 1;
#pragma unroll 1
                    for (int base = 0; base < nr; base += T_) {
#pragma unroll
                        for (int v = 0; v < T_; ++v) {
                            if (base + v < nr) {
                                ring[v] = *ra;
                                if (FB) mir[v] = *rb;
                                ra += RS;
                                rb += RS;
                                if (base + v >= T_ - 1) {
                                    float2 h = make_float2(ring[0].x, ring[0].y), l = make_float2(ring[0].z, ring[0].w);
#pragma unroll
                                    for (int w = 1; w < T_; ++w) ff_add(h, l, ring[w]);
                                    if (FB) {
#pragma unroll
                                        for (int w = 0; w < T_; ++w) ff_add(h, l, mir[w]);
                                    }
                                    put(h, l);
                                }
                            }
                        }
                    }
                } else {
#pragma unroll 1
                    for (int p = 0; p < sp; ++p) {
                        float2 h = make_float2(0.f, 0.f), l = h;
#pragma unroll 4
                        for (int t = 0; t < T; ++t) {
                            ff_add(h, l, ra[(size_t)t * RS]);
                            if (FB) ff_add(h, l, rb[(size_t)t * RS]);
                        }
                        ra += RS;
                        rb += RS;
                        put(h, l);
                    }
                }
            }
            __syncthreads();   // the readers of the rows' sums and of the samples are done
        }
        // the loading, d tr(R)/L (getCaponC.pyx:257-262) or absolute
        for (int p = tid; p < np; p += kCovThreads) {
            float h = 0.f, l = 0.f;
            for (int t = 0; t < T; ++t) {
                const float2 a = tr[p + t];
                const float s = h + a.x, b = s - h;
                l += (h - (s - b)) + (a.x - b) + a.y;
                h = s;
            }
            work[(pix0 + p) * rec + Record::loading(L)].x =
                f.loading == COS_CAPON_LOAD_ABSOLUTE ? f.d * (float)(Ns * T) : f.d * (h + l) / (float)L;
        }
    }
}

// R of the records plus the loading, in the caller's layout
__global__ void general_format_r_kernel(long long n, int L, float scale, int ref_layout,
                                        const float2 *__restrict__ work, float2 *__restrict__ out)
{
    const long long L2 = (long long)L * L;
    const int rec = Record::size(L);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n * L2;
         i += (long long)gridDim.x * blockDim.x) {
        const float2 *const r = work + (i / L2) * rec;
        const int e = (int)(i % L2), a = ref_layout ? e % L : e / L, b = ref_layout ? e / L : e % L;   // element (a, b)
        const int k = min(a, b), d = max(a, b) - k;
        float2 v = r[Record::row(k, L) + d];
        if (a > b) v = cconj(v);
        if (d == 0) v = make_float2(v.x + r[Record::loading(L)].x, 0.f);
        out[i] = cscale(v, scale);
    }
}

// Tile and pairs of a frame, by an estimate of a unit's cycles: the threads' passes
// over the rows' sums (a step costs 16 packed operations) and over the window sums
// (8 a row and entry), counted between whole passes and full lanes since the other
// CTA of an SM fills part of the gaps, and a fixed part a chunk and a unit; times the
// waves of units.  More pairs at a time save barriers; fewer leave room for more
// rows, so that the 2K rows between two tiles are shared by more pixels.  One CTA an
// SM runs a unit in 0.7 of the time of two.  Against the fastest of some 200 measured
// shapes each, for nine frames of L = 7 to 63 and K = 0 to 4, the choice is at most
// 4 % slower.  tile 0: none fits.
CovShape cov_shape(const FrameDev &f, int num_sms)
{
    const int T = 2 * f.K + 1, Ns = f.M - f.L + 1, half = (f.L + 1) / 2, sides = f.fb ? 2 : 1;
    const long long npix = (long long)f.Nx * f.Npy;
    const double threads = kCovThreads;
    CovShape best(0, 1, f.K, f.M, f.L);
    double least = 0;
    for (int per_sm = 2; per_sm >= 1; --per_sm) {
        const size_t room = per_sm == 2 ? 112 * 1024 : 226 * 1024;
        for (int parts : {1, 2, 3, 4, 6, 8, kCovParts}) {
            const int pairs = (half + parts - 1) / parts, chunks = (half + pairs - 1) / pairs;
            const size_t one = CovShape(1, pairs, f.K, f.M, f.L).total, two = CovShape(2, pairs, f.K, f.M, f.L).total;
            if (one > room) continue;
            int tile = (int)std::min<long long>(std::min<long long>(64, f.Npy), npix / num_sms + 1);
            tile = (int)std::min<size_t>(tile, 1 + (room - one) / (two - one + 16));
            while (tile >= 1) {
                CovShape S(tile, pairs, f.K, f.M, f.L);
                const double full = 2.0 * S.rows * pairs / threads, passes = std::ceil(full);
                // items along the tile: the count that keeps the threads fullest
                const double entries = (double)(pairs * (f.L + 1) / sides);
                double window = 0;
                for (int ns = 1; ns <= tile && ns <= 16; ++ns) {
                    const int seg = (tile + ns - 1) / ns;
                    const double n = entries * ns / threads;
                    const double c = (0.3 * std::ceil(n) + 0.7 * n) * (seg * (16.0 * T * sides + 8) + (seg + T) * 4.0 * sides);
                    if (ns == 1 || c < window) {
                        window = c;
                        S.seg = seg;
                        S.nseg = (tile + seg - 1) / seg;
                    }
                }
                const double unit = chunks * ((0.3 * passes + 0.7 * full) * 32.0 * (Ns + f.L) + window + 800.0) + 1000.0 +
                                    (double)S.rows * f.M / 32;
                const long long units = (long long)f.Nx * ((f.Npy + tile - 1) / tile), slots = (long long)num_sms * per_sm;
                const double cost = unit * (per_sm == 2 ? 1.0 : 0.7) * (units <= slots ? 1.0 : (double)units / slots);
                if (best.tile == 0 || cost < least) {
                    best = S;
                    least = cost;
                }
                // the next tile that takes a pass less
                tile = (int)(passes - 1) * kCovThreads / (2 * pairs) - 2 * f.K;
            }
        }
    }
    return best;
}

template <bool FB>
auto cov_pick(int T)
{
    return T == 1   ? cov_kernel<1, FB>
           : T == 3 ? cov_kernel<3, FB>
           : T == 5 ? cov_kernel<5, FB>
           : T == 7 ? cov_kernel<7, FB>
                    : cov_kernel<0, FB>;
}

}  // namespace

// the sizes served are the precise pipeline's (its four warps' sample windows in
// shared memory), within them whatever a tile of one pixel fits
bool general_supported(const FrameDev &f)
{
    if (f.L > 64 || f.refine || (size_t)4 * (2 * f.K + 1) * f.M * sizeof(float2) > 227 * 1024) return false;
    // the fewest pairs that cov_shape tries
    return CovShape(1, ((f.L + 1) / 2 + kCovParts - 1) / kCovParts, f.K, f.M, f.L).total <= 226 * 1024;
}

size_t general_bytes(const FrameDev &f) { return (size_t)f.Nx * f.Npy * Record::size(f.L) * sizeof(float2); }

int launch_general(const FrameDev &f, float2 *work, unsigned *status, int num_sms, cudaStream_t s)
{
    const CovShape S = cov_shape(f, num_sms);
    if (S.tile < 1) return cudaErrorNotSupported;
    const long long units = (long long)f.Nx * ((f.Npy + S.tile - 1) / S.tile);
    if (units > 0x7fffffffLL - 65536) return cudaErrorInvalidValue;
    auto kern = f.fb ? cov_pick<true>(2 * f.K + 1) : cov_pick<false>(2 * f.K + 1);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S.total);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kCovThreads, S.total);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorNotSupported;
    const long long grid = std::min<long long>(units, (long long)num_sms * per_sm);
    kern<<<(unsigned)grid, kCovThreads, S.total, s>>>(f, S, work, (int)units);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const int L = f.L;
    GeneralSolve *solve = L <= 8    ? (f.w ? general_solve_l8_w : general_solve_l8_zp)
                          : L <= 16 ? (f.w ? general_solve_l16_w : general_solve_l16_zp)
                          : L <= 24 ? (f.w ? general_solve_l24_w : general_solve_l24_zp)
                          : L <= 32 ? (f.w ? general_solve_l32_w : general_solve_l32_zp)
                          : L <= 48 ? (f.w ? general_solve_l48_w : general_solve_l48_zp)
                                    : (f.w ? general_solve_l64_w : general_solve_l64_zp);
    if (int r = solve(f, work, status, num_sms, s)) return r;
    if (!f.R) return 0;
    const long long npix = (long long)f.Nx * f.Npy;
    const int ref = f.r_layout == COS_CAPON_R_REFERENCE;
    const float scale = ref ? 1.f : 1.f / ((float)(f.M - L + 1) * (float)(2 * f.K + 1));
    const long long blocks = std::min<long long>((npix * L * L + 255) / 256, (long long)num_sms * 64);
    general_format_r_kernel<<<(unsigned)blocks, 256, 0, s>>>(npix, L, scale, ref, work, f.R);
    return cudaGetLastError();
}

}  // namespace cgb
