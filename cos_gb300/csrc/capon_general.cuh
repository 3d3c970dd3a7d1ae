// Solve stage of the general element-space path (capon_general.cu): FP32
// Cholesky of one pixel's covariance in registers, for any L <= LP.
//
// A pixel's covariance, subarray means and loading are one contiguous record
// in HBM/L2 (Record).  Each warp brings its next pixels' records into its own
// part of shared memory by bulk copies, issued as soon as the current ones are
// in registers, so that the loads (4 KB a pixel at L = 32) ride under a whole
// factorisation; read straight into registers they were exposed between two
// factorisations, since a warp's triangle leaves no room to load ahead.
//
// G lanes own one pixel, lane r the columns j = m*G + r of the upper triangle
// (m < LP/G), the right-hand sides carried along, a pivot row broadcast through
// shared memory.  Two factorisations (matrixDecompc.pyx:19-50), by the subarray length:
//   LP <= 16  that of the fused kernels, R = L D L^H: rows broadcast as they are and
//             scaled by their readers, a product subtracted by two fmas;
//   above     R = U^H U: rows scaled by the pivot's inverse square root before they
//             are broadcast, a product formed and then subtracted.
// The first is faster (65 k pixels, L = 32, z and P: 0.17 ms, 0.20 by the second; 60 k
// pixels, L = 24, weights: 0.12 and 0.15), but rounds twice at the entry's size, and its
// update carries the rounding of the multipliers, which a factor used on both sides
// does not.  Against 64 bits, as a multiple of the precise pipeline's error: w 0.80,
// 0.94, 1.03, 1.04, 1.10, 1.16, 1.27 at L = 5, 16, 20, 24, 32, 40, 64 by the first, 0.92,
// 0.95, 0.99, 0.99, 0.99, 1.01, 1.01 by the second, P alike.  A subarray length between two
// instantiations is padded in front: rows and columns 0 .. pad-1 (pad = LP - L)
// are an identity with zero right-hand sides, and the unrolled steps of those
// rows are skipped, so that padding costs idle column slots only -- the steps
// and trailing rows that run are all real ones.  (Padded behind, every step
// would still update the rows below L.)
#pragma once
#include "capon_common.cuh"
#include "capon_fused_wide.cuh"
#include "capon_internal.h"
#include "capon_tma.cuh"

namespace cgb {
namespace general {

// a pixel's record, in float2 units: the rows k of the upper triangle of R
// (not normalised, not loaded), entries j - k = 0 .. L-1-k, each row padded to
// 16 bytes; the L subarray means; the loading in the last pair's first word
struct Record {
    __host__ __device__ static int row(int k, int L)
    {
        return k * L - k * (k - 1) / 2 + ((L & 1) ? (k + 1) / 2 : k / 2);
    }
    __host__ __device__ static int mean(int L) { return row(L, L); }
    __host__ __device__ static int loading(int L) { return mean(L) + ((L + 1) & ~1); }
    __host__ __device__ static int size(int L) { return loading(L) + 2; }
};

// WARPS and BLOCKS (resident CTAs an SM): as many warps as the register
// triangle of LP columns leaves room for
template <int LP_, int G_, int MAXPAD_, int WARPS_, int BLOCKS_>
struct SolveCfg {
    static constexpr int LP = LP_, G = G_, MAXPAD = MAXPAD_;  // pad < MAXPAD
    static constexpr int WARPS = WARPS_, BLOCKS = BLOCKS_;
    static constexpr int NM = LP / G, PPW = 32 / G;
    static constexpr bool LDL = LP <= 16;   // R = L D L^H, else U^H U
    // float4 slots of a pixel's shared area: two pivot rows, or the exchange
    // area of the back substitution
    static constexpr int RB = 2 * (LP + 1), XCH = (G * (G + 1) + 1) / 2;
    static constexpr int AREA = RB > XCH ? RB : XCH;
    static constexpr size_t BAR = 128;  // a barrier per warp
    static size_t smem(int L)
    {
        return BAR + (size_t)WARPS * PPW * (AREA * sizeof(float4) + Record::size(L) * sizeof(float2));
    }
};

// W: the weights are wanted (one right-hand side and a back substitution, as
// the fused w mode); otherwise z and P from the two right-hand sides
template <class C, bool W>
__global__ void __launch_bounds__(32 * C::WARPS, C::BLOCKS)
solve_kernel(FrameDev f, const float2 *__restrict__ work, long long npix, unsigned *status)
{
    constexpr int LP = C::LP, G = C::G, NM = C::NM, PPW = C::PPW;
    extern __shared__ __align__(128) unsigned char smraw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gi = lane / G, r = lane % G;
    const int L = f.L, pad = LP - L, rec = Record::size(L);
    uint64_t *const bar = (uint64_t *)smraw + warp;
    float4 *const rb = (float4 *)(smraw + C::BAR) + (size_t)(warp * PPW + gi) * C::AREA;
    float2 *const in = (float2 *)(smraw + C::BAR + (size_t)C::WARPS * PPW * C::AREA * sizeof(float4)) +
                       (size_t)warp * PPW * rec;
    const float nt = (float)(f.M - L + 1) * (float)(2 * f.K + 1);
    const float2 zero = make_float2(0.f, 0.f);
    const long long step = (long long)gridDim.x * C::WARPS * PPW;
    long long p0 = ((long long)blockIdx.x * C::WARPS + warp) * PPW;
    // lane 0: the records of pixels p .. p+PPW-1 (the last one again past the end)
    auto issue = [&](long long p) {
        fused::fence_proxy_async();
        fused::mbar_expect_tx(bar, (uint32_t)(PPW * rec * sizeof(float2)));
        for (int q = 0; q < PPW; ++q) {
            const long long pix = p + q < npix ? p + q : npix - 1;
            fused::bulk_g2s(in + q * rec, work + (size_t)pix * rec, (uint32_t)(rec * sizeof(float2)), bar);
        }
    };
    if (lane == 0) {
        fused::mbar_init(bar, 1);
        fused::fence_mbar_init();
        if (p0 < npix) issue(p0);
    }
    __syncwarp();
    uint32_t phase = 0;
#pragma unroll 1
    for (; p0 < npix; p0 += step, phase ^= 1u) {
        const bool active = p0 + gi < npix;
        const long long pix = active ? p0 + gi : npix - 1;
        if (!__all_sync(0xffffffffu, fused::mbar_wait_bounded(bar, phase))) {
            if (lane == 0) {
                atomicOr(status, ERR_TIMEOUT);
                fused::mbar_wait_bounded(bar, phase);  // let the copies land before the CTA leaves
            }
            return;
        }
        const float2 *const R = in + gi * rec;
        const float dl = R[Record::loading(L)].x;
        float2 A[LP][NM], b1[NM], b2[NM];
        float dinv[NM];
        // row k (padded index) at Rk[j], advanced row by row
        const float2 *Rk = R + r;
        fused::static_for<0, LP>([&](auto kc) __attribute__((always_inline)) {
            constexpr int k = decltype(kc)::value, mk = k / G;
            const bool real = k >= C::MAXPAD || k >= pad;
#pragma unroll
            for (int m = mk; m < NM; ++m) {
                float2 v = make_float2(0.f, 0.f);
                if (real && (m > mk || r >= k % G)) v = Rk[m * G - k];
                A[k][m] = v;
            }
            // the loading on the diagonal; 1 on the padding's
            if (r == k % G) A[k][mk] = make_float2(real ? A[k][mk].x + dl : 1.f, 0.f);
            if (real) Rk += (LP - k + 1) & ~1;
        });
#pragma unroll
        for (int m = 0; m < NM; ++m) {
            const int j = m * G + r;
            b1[m] = make_float2(j >= pad ? 1.f : 0.f, 0.f);
            b2[m] = j >= pad ? R[Record::mean(L) + j - pad] : make_float2(0.f, 0.f);
            dinv[m] = 1.f;
        }
        __syncwarp();
        if (lane == 0 && p0 + step < npix) issue(p0 + step);
        bool bad = false;
        float s11 = 0.f, s11l = 0.f;  // high part and the sum of its rounding errors
        float2 s12 = make_float2(0.f, 0.f);
        // row `row` as (-Re, +Im, -Im, -Re) of A[row][j]; slot LP carries the row's
        // right-hand sides.  U^H U: all of them by the pivot's inverse square root first
        auto publish = [&](auto rc, float4 *buf) __attribute__((always_inline)) {
            constexpr int row = decltype(rc)::value, mrow = row / G;
            if constexpr (!C::LDL) {
                const float dv = __shfl_sync(0xffffffffu, A[row][mrow].x, row % G, G);
                bad |= !(dv > 0.f);
                // the unit's approximation and one Newton step: its error is common to the
                // whole row
                const float y0 = rsqrtf(dv), inv = fmaf(0.5f * y0, fmaf(-dv * y0, y0, 1.f), y0);
#pragma unroll
                for (int m = mrow; m < NM; ++m) A[row][m] = cscale(A[row][m], inv);
                if (r == row % G) {
                    if (W) dinv[mrow] = inv;
                    b1[mrow] = cscale(b1[mrow], inv);
                    if (!W) b2[mrow] = cscale(b2[mrow], inv);
                }
            }
#pragma unroll
            for (int m = mrow; m < NM; ++m)
                buf[m * G + r] = make_float4(-A[row][m].x, A[row][m].y, -A[row][m].y, -A[row][m].x);
            if (r == row % G)
                buf[LP] = make_float4(b1[mrow].x, b1[mrow].y, W ? 0.f : b2[mrow].x, W ? 0.f : b2[mrow].y);
        };
        __syncwarp();  // the area's readers of the last pixel are done
        if (pad == 0) publish(std::integral_constant<int, 0>{}, rb);
        fused::static_for<0, LP>([&](auto ic) __attribute__((always_inline)) {
            constexpr int i = decltype(ic)::value, oi = i % G, mi = i / G;
            float4 *const nxt = rb + ((i + 1) & 1) * (LP + 1);
            if (i < C::MAXPAD && i < pad) {
                // a padding row: nothing to eliminate
                if constexpr (i + 1 < LP)
                    if (i + 1 == pad) publish(std::integral_constant<int, i + 1>{}, nxt);
            } else {
                // step i reads buffer i & 1, written at step i-1 and last read
                // at step i-2, before the barrier that ended step i-1
                float4 *const rbi = rb + (i & 1) * (LP + 1);
                __syncwarp();
                const float4 yy = rbi[LP];
                // rdv scales the row and its right-hand sides at the reader (L D L^H)
                float rdv = 1.f;
                if constexpr (C::LDL) {
                    const float dv = -rbi[i].x;
                    bad |= !(dv > 0.f);
                    rdv = __frcp_rn(dv);
                    if (W && r == oi) dinv[mi] = rdv;
                }
                auto scaled = [&](float v) { return C::LDL ? v * rdv : v; };
                const float2 y1 = make_float2(scaled(yy.x), scaled(yy.y)), y2 = make_float2(scaled(yy.z), scaled(yy.w));
                {
                    const float t = fmaf(yy.x, y1.x, yy.y * y1.y), s = s11 + t;
                    s11l += t - (s - s11);
                    s11 = s;
                }
                if (!W) s12 = cadd(s12, cconjmul(make_float2(yy.x, yy.y), y2));
                const float2 y1s = make_float2(y1.y, y1.x), y2s = make_float2(y2.y, y2.x);
                // c + b d + a e, the sum of products first or two fmas
                auto update = [&](float2 a, float2 e, float2 b, float2 d, float2 c) __attribute__((always_inline)) {
                    return C::LDL ? ffma2(a, e, ffma2(b, d, c)) : fadd2(c, ffma2(a, e, ffma2(b, d, zero)));
                };
                float2 vrr[NM], vii[NM];
#pragma unroll
                for (int m = mi; m < NM; ++m) {
                    const float2 v = A[i][m];
                    const float2 n1 = make_float2(-v.x, -v.x), n2 = make_float2(-v.y, v.y);
                    const float2 t1 = update(n2, y1s, n1, y1, b1[m]);
                    const bool below = m > mi || r > oi;
                    if (below) b1[m] = t1;
                    if (!W) {
                        const float2 t2 = update(n2, y2s, n1, y2, b2[m]);
                        if (below) b2[m] = t2;
                    }
                    const float vr = scaled(v.x), vi = scaled(v.y);
                    vrr[m] = make_float2(vr, vr);
                    vii[m] = make_float2(vi, vi);
                }
                // row i+1 first, published before the bulk of the update
#pragma unroll
                for (int k = i + 1; k < LP; ++k) {
                    const float4 u4 = rbi[k];
#pragma unroll
                    for (int m = mi; m < NM; ++m)
                        if (m >= k / G)
                            A[k][m] = update(vii[m], make_float2(u4.z, u4.w), vrr[m], make_float2(u4.x, u4.y), A[k][m]);
                    if constexpr (i + 1 < LP)
                        if (k == i + 1) publish(std::integral_constant<int, i + 1>{}, nxt);
                }
            }
        });
        // a non-positive pivot leaves no Cholesky factor: not finite, as a
        // square root of it would be
        const float is11 = bad ? __int_as_float(0x7fc00000) : 1.0f / (s11 + s11l);
        if (active && r == 0) {
            if (!W) f.z[pix] = make_float2(s12.x * is11, s12.y * is11);
            if (f.P) f.P[pix] = is11 / nt;
            if (bad) atomicOr(status, ERR_NOT_PD);
        }
        if constexpr (W) {
            // (D L^H) x = b1, or U x = b1, by blocks of G rows, last block first, through the
            // exchange area (the fused w mode's scheme, capon_fused.cuh)
            float2 xv[NM];
#pragma unroll
            for (int m = 0; m < NM; ++m) xv[m] = make_float2(0.f, 0.f);
            float2 *const X = (float2 *)rb;
            __syncwarp();
#pragma unroll
            for (int m = NM - 1; m >= 0; --m) {
#pragma unroll
                for (int q = 0; q < G; ++q) {
                    float2 e = make_float2(0.f, 0.f);
#pragma unroll
                    for (int mm = m + 1; mm < NM; ++mm) e = cadd(e, cmul(A[m * G + q][mm], xv[mm]));
                    X[q * (G + 1) + r] = e;
                }
                __syncwarp();
                float2 acc = b1[m];
#pragma unroll 1
                for (int l = 0; l < G; ++l) acc = csub(acc, X[r * (G + 1) + l]);
                __syncwarp();
#pragma unroll
                for (int q = 0; q < G; ++q) X[q * (G + 1) + r] = A[m * G + q][m];
                __syncwarp();
                float2 xm = xv[m];
#pragma unroll 1
                for (int q = G - 1; q >= 0; --q) {
                    const float2 xq = shfl2(cscale(acc, dinv[m]), q, G);
                    if (r == q) xm = xq;
                    const float2 t = csub(acc, cmul(X[r * (G + 1) + q], xq));
                    acc = make_float2(r < q ? t.x : acc.x, r < q ? t.y : acc.y);
                }
                xv[m] = xm;
                __syncwarp();
            }
            // w = x / sum(x): by the sum of the x at hand, so that the weights sum to one
            // to rounding, as 1/s11 of the forward pass would leave them only to the
            // error of x (2e-6 at L = 63)
            float2 zp = make_float2(0.f, 0.f), sum = zp;
#pragma unroll
            for (int m = 0; m < NM; ++m) {
                const float2 t = cconjmul(xv[m], b2[m]);
                if (m * G + r >= pad) {
                    zp = cadd(zp, t);
                    sum = cadd(sum, xv[m]);
                }
            }
#pragma unroll
            for (int o = G / 2; o; o >>= 1) {
                zp = cadd(zp, shfl2_xor(zp, o, G));
                sum = cadd(sum, shfl2_xor(sum, o, G));
            }
            const float den = cabs2(sum);
            const float2 isum = bad ? make_float2(is11, is11) : make_float2(sum.x / den, -sum.y / den);
            if (active && r == 0) f.z[pix] = cmul(zp, cconj(isum));
            if (active && f.w) {
#pragma unroll
                for (int m = 0; m < NM; ++m)
                    if (m * G + r >= pad) f.w[(size_t)pix * L + m * G + r - pad] = cmul(xv[m], isum);
            }
        }
    }
}

template <class C, bool W>
int launch_solve(const FrameDev &f, const float2 *work, unsigned *status, int num_sms, cudaStream_t s)
{
    const long long npix = (long long)f.Nx * f.Npy, per_block = C::WARPS * C::PPW;
    const long long groups = (npix + per_block - 1) / per_block;
    const size_t smem = C::smem(f.L);
    auto kern = solve_kernel<C, W>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * C::WARPS, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorNotSupported;
    const long long most = (long long)num_sms * per_sm;
    kern<<<(unsigned)(groups < most ? groups : most), 32 * C::WARPS, smem, s>>>(f, work, npix, status);
    return cudaGetLastError();
}

}  // namespace general
}  // namespace cgb
