// General element-space path for sm_103a: z, P and w for the frames without a
// fused instantiation -- any subarray length L <= 64, any window, and
// forward-backward averaging.
//
//   1. covariance kernel (this file): R per pixel, float-float sums of FP32
//      window products, rounded once, to HBM/L2 as the solve stage's records;
//   2. solve kernel (capon_general.cuh): FP32 Cholesky in registers and the
//      outputs.
//
// Covariance.  Along diagonal d,
//   R[k,k+d] = sum_{i=k}^{k+Ns-1} q_d[i],   q_d[i] = sum_{t<T} x_t[i] conj(x_t[i+d]),
// (the smoothing and temporal averaging of getCaponC.pyx:197-242 with the sums
// exchanged).  The precise pipeline formed the T Ns L products of every
// pixel's first row and 2 T more per entry below it from shared memory, one
// lane per diagonal.  Here each product x_y[i] conj(x_y[i+d]) of a range row is
// formed once for all the pixels whose window holds the row:
//   products  a thread owns a 4 x 2 block of (i, d) and walks the rows of the
//             tile with the last T row products in registers, so a row costs 9
//             sample loads for 8 products and a pixel T - 1 additions; the
//             sums q go to shared memory;
//   diagonals a thread per (pixel, d) sums q_d[0..Ns-1] and slides along the
//             diagonal, R[k] = R[k-1] + q[k-1+Ns] - q[k-1], all in float-float
//             (TwoSum).  q itself is one FP32 sum of T products, so R is the
//             exactly accumulated sum of the same q everywhere, rounded once.
//             (Differences q[k-1+Ns] - q[k-1] and pairs of q rounded to FP32
//             first would save a third of these operations, but their errors
//             add up along a diagonal: P against 64 bits twice as far off where
//             the window has fewer snapshots than L.)
//             Forward-backward averaging, (R + J R^T J)/2, pairs row k with
//             row L-1-d-k of the same diagonal, which is the sliding sum over
//             the mean of q_d[i] and q_d[M-1-d-i].
// What bounds it: issue (48 %) with waits at the barriers between the phases,
// whose threads two CTAs an SM only partly fill (6 pixels x 32 diagonals of 256
// threads at M=64, L=32); DRAM traffic is the cube read and the records written
// once.  Measured, 60 k pixels at M=48, L=24, K=2 with weights: 1.44 ms in the
// precise pipeline, 0.17 ms here + 0.12 ms in the solve stage; 65 k pixels at
// M=64, L=32, K=2 with forward-backward averaging: 2.56 ms, 0.38 + 0.17 ms.
#include <algorithm>
#include <type_traits>

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
constexpr int kCovMaxM = 1020;       // i / 4 fits a byte of the block table

struct CovShape {
    int tile;        // pixels per unit
    int seg, nseg;   // pixels per product item, items along the tile
    int XS, LS;      // sample row stride; row stride of q up to row Ns - 1
    int QS;          // entries of q a pixel holds
    int EB;          // bytes of an entry: 8, or 16 for the exact form (value and remainder)
    int blocks;      // (i, d) blocks that hold an entry
    size_t off_q, off_tab, off_row, total;
    __host__ __device__ CovShape(int tile_, int K, int M, int L, bool exact)
    {
        tile = tile_;
        EB = exact ? 16 : 8;
        seg = tile;
        nseg = 1;
        LS = (L + 1) & ~1;
        QS = row(M, M, L);
        XS = (M + 6 + 1) & ~1;  // a block reads up to 5 samples past its last valid column
        blocks = 0;
        for (int i = 0; i < M; i += 4) blocks += cols(i, M);
        off_q = (size_t)(tile + 2 * K) * XS * sizeof(float2);
        // LS entries past the last pixel's: lanes past a diagonal's end read on
        off_tab = off_q + ((size_t)tile * QS + LS) * EB;
        off_row = off_tab + (((size_t)blocks * sizeof(unsigned short) + 15) & ~(size_t)15);
        total = off_row + (((size_t)(M + 4) * sizeof(int) + 15) & ~(size_t)15);
    }
    // offset of row i of q: LS entries up to row Ns - 1, then as many as the row
    // holds (i + d < M), rounded up to pairs
    __host__ __device__ int row(int i, int M, int L) const
    {
        const int Ns = M - L + 1;
        return i <= Ns ? i * LS : Ns * LS + Record::row(i - Ns, L - 1);
    }
    // 2-column blocks of the rows i .. i+3 that hold an entry i + d < M
    __host__ __device__ int cols(int i, int M) const { return LS / 2 < (M - i + 1) / 2 ? LS / 2 : (M - i + 1) / 2; }
};

// i / d by the reciprocal of d; exact while the quotient times d stays below 2^21
COS_DEV int small_div(int i, float inv) { return (int)(((float)i + 0.5f) * inv); }

// x_y[i0+a] conj(x_y[i0+d0+a+b]) for a < 4, b < 2 as out[2a+b] += / =
template <bool ACC>
COS_DEV void block_products(float2 (&out)[8], const float2 *xi, const float2 *xj)
{
    const float4 a01 = *(const float4 *)xi, a23 = *(const float4 *)(xi + 2);
    const float4 c01 = *(const float4 *)xj, c23 = *(const float4 *)(xj + 2);
    const float2 c4 = xj[4];
    const float2 a[4] = {make_float2(a01.x, a01.y), make_float2(a01.z, a01.w), make_float2(a23.x, a23.y),
                         make_float2(a23.z, a23.w)};
    const float2 c[5] = {make_float2(c01.x, c01.y), make_float2(c01.z, c01.w), make_float2(c23.x, c23.y),
                         make_float2(c23.z, c23.w), c4};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 as = make_float2(a[q].y, -a[q].x);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const float2 v = c[q + b], z = ACC ? out[2 * q + b] : make_float2(0.f, 0.f);
            // a conj(c) = c.re (ar, ai) + c.im (ai, -ar)
            out[2 * q + b] = ffma2(make_float2(v.y, v.y), as, ffma2(make_float2(v.x, v.x), a[q], z));
        }
    }
}

// the same added to the float-float (h, l), every product exact (TwoProd by fma)
COS_DEV void block_products_exact(float2 (&h)[8], float2 (&l)[8], const float2 *xi, const float2 *xj)
{
    const float2 z = make_float2(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 a = xi[q], as = make_float2(a.y, -a.x);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const float2 v = xj[q + b], vr = make_float2(v.x, v.x), vi = make_float2(v.y, v.y);
            const float2 p1 = ffma2(vr, a, z), p2 = ffma2(vi, as, z);
            const float2 e1 = ffma2(vr, a, make_float2(-p1.x, -p1.y)), e2 = ffma2(vi, as, make_float2(-p2.x, -p2.y));
            two_sum_acc(h[2 * q + b], l[2 * q + b], p1);
            two_sum_acc(h[2 * q + b], l[2 * q + b], p2);
            l[2 * q + b] = fadd2(l[2 * q + b], fadd2(e1, e2));
        }
    }
}

// T: the temporal window 2K+1, 0 = taken from the frame (products formed anew
// for every pixel of the window: the row ring needs a compile-time length).
// EXACT (T = 0): q and everything after it in float-float, the products exact.
template <int T_, bool FB, bool EXACT = false>
__global__ void __launch_bounds__(kCovThreads, 2)
cov_kernel(FrameDev f, CovShape S, float2 *__restrict__ work, int units)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const int M = f.M, L = f.L, K = T_ ? (T_ - 1) / 2 : f.K, T = 2 * K + 1, Ns = M - L + 1;
    const int XS = S.XS, LS = S.LS, QS = S.QS, tid = threadIdx.x, rec = Record::size(L);
    float2 *xs = (float2 *)smraw;
    static_assert(!EXACT || T_ == 0, "the exact form takes any window");
    using Entry = typename std::conditional<EXACT, float4, float2>::type;   // (value, remainder) or the value
    Entry *qs = (Entry *)(smraw + S.off_q);
    unsigned short *tab = (unsigned short *)(smraw + S.off_tab);
    int *rowq = (int *)(smraw + S.off_row);   // offsets of the rows of q
    for (int i = tid; i < M; i += kCovThreads) rowq[i] = S.row(i, M, L);
    // the (i, d) blocks, dense: (i/4) << 8 | d/2
    for (int t = tid; t < (M + 3) / 4 * (LS / 2); t += kCovThreads) {
        const int a = t / (LS / 2), b = t % (LS / 2);
        if (b >= S.cols(4 * a, M)) continue;
        int off = b;
        for (int u = 0; u < a; ++u) off += S.cols(4 * u, M);
        tab[off] = (unsigned short)(a << 8 | b);
    }
    const int tiles_per_beam = (f.Npy + S.tile - 1) / S.tile;
    const float inv_blocks = 1.f / (float)S.blocks, inv_L = 1.f / (float)L, inv_M = 1.f / (float)M;
#pragma unroll 1
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
        const int bx = u / tiles_per_beam, p0 = (u % tiles_per_beam) * S.tile;
        const int np = min(S.tile, f.Npy - p0), rows = np + 2 * K;
        const size_t pix0 = (size_t)bx * f.Npy + p0;
        const float2 *src = f.x + ((size_t)bx * f.Ny + p0) * M;
        __syncthreads();  // the last unit's readers are done
        for (int i = tid; i < rows * M; i += kCovThreads) {
            const int r = small_div(i, inv_M);
            xs[r * XS + (i - r * M)] = src[i];
        }
        for (int i = tid; i < rows * (XS - M); i += kCovThreads) {
            const int r = i / (XS - M);
            xs[r * XS + M + (i - r * (XS - M))] = make_float2(0.f, 0.f);
        }
        __syncthreads();

        // ---- products: window sums q of the tile's pixels
#pragma unroll 1
        for (int it = tid; it < S.blocks * S.nseg; it += kCovThreads) {
            const int sg = small_div(it, inv_blocks), e = tab[it - sg * S.blocks];
            const int i0 = (e >> 8) * 4, d0 = (e & 255) * 2, s0 = sg * S.seg, sp = min(S.seg, np - s0);
            const float2 *xi = xs + s0 * XS + i0, *xj = xi + d0;
            Entry *qd = qs + (size_t)s0 * QS + d0;
            int ro[4];   // -1: the row has no entry in these columns
#pragma unroll
            for (int a = 0; a < 4; ++a) ro[a] = i0 + a + d0 < M ? rowq[i0 + a] : -1;
            auto put = [&](const float2(&v)[8]) __attribute__((always_inline)) {
#pragma unroll
                for (int a = 0; a < 4; ++a)
                    if (ro[a] >= 0)
                        *(float4 *)(qd + ro[a]) = make_float4(v[2 * a].x, v[2 * a].y, v[2 * a + 1].x, v[2 * a + 1].y);
                qd += QS;
            };
            if constexpr (EXACT) {
#pragma unroll 1
                for (int p = 0; p < sp; ++p) {
                    float2 h[8], l[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) h[q] = l[q] = make_float2(0.f, 0.f);
#pragma unroll 1
                    for (int t = 0; t < T; ++t) block_products_exact(h, l, xi + (p + t) * XS, xj + (p + t) * XS);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float2 v = fadd2(h[q], l[q]), e = fsub2(l[q], fsub2(v, h[q]));
                        if (ro[q / 2] >= 0) qd[ro[q / 2] + q % 2] = make_float4(v.x, v.y, e.x, e.y);
                    }
                    qd += QS;
                }
            } else if constexpr (T_ != 0) {
                float2 ring[T_][8];
                const int nr = sp + T_ - 1;
#pragma unroll 1
                for (int base = 0; base < nr; base += T_) {
#pragma unroll
                    for (int v = 0; v < T_; ++v) {
                        if (base + v < nr) {
                            block_products<false>(ring[v], xi, xj);
                            xi += XS;
                            xj += XS;
                            if (base + v >= T_ - 1) {
                                float2 sum[8];
#pragma unroll
                                for (int q = 0; q < 8; ++q) {
                                    sum[q] = ring[0][q];
#pragma unroll
                                    for (int w = 1; w < T_; ++w) sum[q] = fadd2(sum[q], ring[w][q]);
                                }
                                put(sum);
                            }
                        }
                    }
                }
            } else {
#pragma unroll 1
                for (int p = 0; p < sp; ++p) {
                    float2 sum[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) sum[q] = make_float2(0.f, 0.f);
#pragma unroll 1
                    for (int t = 0; t < T; ++t) block_products<true>(sum, xi + (p + t) * XS, xj + (p + t) * XS);
                    put(sum);
                }
            }
        }
        // subarray means of the centre rows, g[l] = (1/Ns) sum_s x[s+l]
        // (getCaponC.pyx:246-255)
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
        __syncthreads();

        // ---- the loading, d tr(R)/L (getCaponC.pyx:257-262) or absolute: a warp
        // per pixel sums tr(R) = sum_i c_i q_0[i] (c_i subarrays hold channel i)
        // in float-float
        for (int p = tid >> 5; p < np; p += kCovThreads / 32) {
            float h = 0.f, l = 0.f;
            for (int i = tid & 31; i < M; i += 32) {
                const Entry e = qs[(size_t)p * QS + rowq[i]];
                const float c = (float)min(min(i + 1, M - i), min(L, Ns)), v = e.x;
                const float pr = c * v, s = h + pr, bb = s - h;
                l += (h - (s - bb)) + (pr - bb) + fmaf(c, v, -pr);
                if constexpr (EXACT) l = fmaf(c, e.z, l);
                h = s;
            }
            for (int o = 16; o; o >>= 1) {
                const float oh = __shfl_xor_sync(0xffffffffu, h, o), ol = __shfl_xor_sync(0xffffffffu, l, o);
                const float s = h + oh, bb = s - h;
                l += (h - (s - bb)) + (oh - bb) + ol;
                h = s;
            }
            if ((tid & 31) == 0)
                work[(pix0 + p) * rec + Record::loading(L)].x =
                    f.loading == COS_CAPON_LOAD_ABSOLUTE ? f.d * (float)(Ns * T) : f.d * (h + l) / (float)L;
        }
        // ---- diagonals.  Every lane runs all L rows, four at a time, so that the
        // loads and the TwoSums of four rows overlap (with the diagonal's own
        // length as the bound, each row waited for the last: 200 cycles); rows
        // past its end read in-bounds leftovers and store nothing
#pragma unroll 1
        for (int it = tid; it < np * L; it += kCovThreads) {
            const int p = small_div(it, inv_L), d = it - p * L, n = L - d;
            const Entry *q = qs + (size_t)p * QS + d;
            float2 *out = work + (pix0 + p) * rec + d;
            if constexpr (EXACT) {
                float2 h = make_float2(0.f, 0.f), l = h;
                // (h, l) += sign times entry i (and its mirror: halved at the store)
                auto add = [&](int i, float sign) __attribute__((always_inline)) {
                    float4 e = q[rowq[i]];
                    two_sum_acc(h, l, make_float2(sign * e.x, sign * e.y));
                    l = fadd2(l, make_float2(sign * e.z, sign * e.w));
                    if (FB) {
                        e = q[rowq[max(M - 1 - d - i, 0)]];
                        two_sum_acc(h, l, make_float2(sign * e.x, sign * e.y));
                        l = fadd2(l, make_float2(sign * e.z, sign * e.w));
                    }
                };
#pragma unroll 2
                for (int i = 0; i < Ns; ++i) add(i, 1.f);
#pragma unroll 2
                for (int k = 0; k < L; ++k) {
                    float2 r = fadd2(h, l);
                    if (FB) r = cscale(r, 0.5f);
                    if (k < n) *out = r;
                    out += (L - k + 1) & ~1;
                    if (k + 1 < L) {
                        add(k + Ns, 1.f);
                        add(k, -1.f);
                    }
                }
            } else {
                // entry i of the diagonal, at offset o; forward-backward: q_d[i] + q_d[M-1-d-i]
                // takes its place, halved at the store
                auto term = [&](int i, int o) __attribute__((always_inline)) {
                    return FB ? fadd2(q[o], q[rowq[max(M - 1 - d - i, 0)]]) : q[o];
                };
                float2 h = make_float2(0.f, 0.f), l = h;
                {
                    // q[0] + .. + q[Ns-1] on two chains
                    float2 h1 = h, l1 = h;
                    int i = 0;
#pragma unroll 4
                    for (; i + 1 < Ns; i += 2) {
                        two_sum_acc(h, l, term(i, i * LS));
                        two_sum_acc(h1, l1, term(i + 1, (i + 1) * LS));
                    }
                    if (i < Ns) two_sum_acc(h, l, term(i, i * LS));
                    two_sum_acc(h, l, h1);
                    l = fadd2(l, l1);
                }
#pragma unroll 1
                for (int k0 = 0; k0 < L; k0 += 4) {
                    float2 add[4], sub[4];
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        // the last row's step is not used
                        const int i = min(k0 + v, max(L - 2, 0)), j = L > 1 ? i + Ns : 0;
                        add[v] = term(j, rowq[j]);
                        sub[v] = term(i, rowq[i]);
                    }
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        float2 r = fadd2(h, l);
                        if (FB) r = cscale(r, 0.5f);
                        if (k0 + v < n) *out = r;
                        out += (L - k0 - v + 1) & ~1;
                        two_sum_acc(h, l, add[v]);
                        two_sum_acc(h, l, make_float2(-sub[v].x, -sub[v].y));
                    }
                }
            }
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

// With few snapshots for the subarray length R is close to singular but for the
// loading, and the rounding of the FP32 products, the same along a diagonal, shows
// in P (L = 34, M = 65, K = 0: more than 1.5 times as far from 64 bits as with
// exact products; at 2.5 L snapshots and more no difference).  Those frames take
// the exact form.
bool exact_form(const FrameDev &f) { return 2 * (2 * f.K + 1) * (f.M - f.L + 1) < 5 * f.L; }

// the tile of a frame: two CTAs an SM where four pixels or more fit so, one
// otherwise; no longer than what leaves every SM a unit.  tile 0: none fits.
CovShape cov_shape(const FrameDev &f, int num_sms)
{
    const int T = 2 * f.K + 1;
    const bool exact = exact_form(f);
    const CovShape one(1, f.K, f.M, f.L, exact);
    if (one.total > 226 * 1024) return CovShape(0, f.K, f.M, f.L, exact);
    const size_t per = (size_t)one.XS * sizeof(float2) + (size_t)one.QS * one.EB;
    auto room = [&](size_t most) {
        return one.total > most ? 0 : 1 + (int)std::min<size_t>(63, (most - one.total) / per);
    };
    int tile = room(112 * 1024);
    if (tile < 4) tile = room(226 * 1024);
    const long long npix = (long long)f.Nx * f.Npy;
    tile = (int)std::min<long long>(std::min(tile, f.Npy), std::max<long long>(1, npix / num_sms));
    // whole passes of the diagonals' threads
    if (const int waves = tile * f.L / kCovThreads) tile = std::min(tile, waves * kCovThreads / f.L);
    CovShape S(tile, f.K, f.M, f.L, exact);
    // product items along the tile: the count that keeps the threads fullest
    long best = -1;
    for (int ns = 1; tile && ns <= tile; ++ns) {
        const int seg = (tile + ns - 1) / ns;
        const long passes = ((long)S.blocks * ns + kCovThreads - 1) / kCovThreads;
        // a row's products and loads cost about 28 cycles, a pixel's sums and stores 8 + 8 (T - 1)
        const long cost = passes * ((long)(seg + T - 1) * 28 + (long)seg * (8 + 8 * (T - 1)));
        if (best < 0 || cost < best) {
            best = cost;
            S.seg = seg;
            S.nseg = (tile + seg - 1) / seg;
        }
    }
    return S;
}

template <bool FB>
auto cov_pick(int T, bool exact)
{
    return exact    ? cov_kernel<0, FB, true>
           : T == 1   ? cov_kernel<1, FB>
           : T == 3 ? cov_kernel<3, FB>
           : T == 5 ? cov_kernel<5, FB>
           : T == 7 ? cov_kernel<7, FB>
                    : cov_kernel<0, FB>;
}

}  // namespace

bool general_supported(const FrameDev &f)
{
    if (f.L > 64 || f.refine) return false;
    const CovShape S(1, f.K, f.M, f.L, exact_form(f));
    return S.total <= 226 * 1024 && f.M <= kCovMaxM;
}

size_t general_bytes(const FrameDev &f) { return (size_t)f.Nx * f.Npy * Record::size(f.L) * sizeof(float2); }

int launch_general(const FrameDev &f, float2 *work, unsigned *status, int num_sms, cudaStream_t s)
{
    const CovShape S = cov_shape(f, num_sms);
    if (S.tile < 1) return cudaErrorNotSupported;
    const long long units = (long long)f.Nx * ((f.Npy + S.tile - 1) / S.tile);
    if (units > 0x7fffffffLL - 65536) return cudaErrorInvalidValue;
    const bool exact = exact_form(f);
    auto kern = f.fb ? cov_pick<true>(2 * f.K + 1, exact) : cov_pick<false>(2 * f.K + 1, exact);
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
