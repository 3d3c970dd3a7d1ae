// General batched solve A x = b (cos_capon_solve / ISolver::solve) for sm_103a:
// Gaussian elimination with partial pivoting by modulus, A column-major as in
// the reference's Solver (testRTC.pyx:227-229 solves A^T x = b on row-major
// input).
//
// A thread owns one row of [A | b] in registers; G lanes (8, 16 or 32, or two or
// three warps past N = 32) own a system.  Rows are never moved: each lane keeps
// the position its row would have after the exchanges, so the pivot choice, ties
// included, is that of the exchanging form.  Step i reduces |a_ri|^2 over the
// rows left, the pivot's owner publishes its row through shared memory, two
// columns a store, and every row left subtracts its multiple with four fmas a
// column (a row published as (re, re, im, im) for two packed fmas a column took
// the one storing lane as long as the update itself: 0.29 ms against 0.19).  The
// back substitution runs the columns from the last, each unknown broadcast from
// its owner.
//
// Before, a warp held the system in shared memory, updated one row at a time (a
// third of the lanes idle on average, two barriers a row) and left the back
// substitution to lane 0: 16,256 systems of N = 32 took 0.48 ms; here 0.19 ms.
// What bounds it: issue (56 %) over the N dependent pivot steps, about 8 k
// instructions a system at N = 32 with half the rows finished on average; a
// system needs 2 N^2 registers over its lanes, which leaves 16 warps an SM.
#include "capon_common.cuh"
#include "capon_fused_wide.cuh"
#include "capon_internal.h"

namespace cgb {
namespace {

// max over the G lanes of a system (G <= 32; all lanes of the warp take part)
template <int G>
COS_DEV unsigned group_max(unsigned v)
{
    if constexpr (G == 32) {
        return __reduce_max_sync(0xffffffffu, v);
    } else {
#pragma unroll
        for (int o = G / 2; o; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o, G));
        return v;
    }
}
template <int G>
COS_DEV unsigned group_min(unsigned v)
{
    if constexpr (G == 32) {
        return __reduce_min_sync(0xffffffffu, v);
    } else {
#pragma unroll
        for (int o = G / 2; o; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o, G));
        return v;
    }
}

// NP: columns held (N <= NP); G: threads per system; THREADS per CTA.  With
// G > 32 a CTA is one system and its warps meet at CTA barriers.
template <int NP, int G, int THREADS>
__global__ void __launch_bounds__(THREADS)
lu_solve_kernel(int N, long long batch, const float2 *__restrict__ Ag, const float2 *__restrict__ bg,
                float2 *__restrict__ xg)
{
    constexpr bool WIDE = G > 32;
    constexpr int PER = THREADS / G, W = WIDE ? G / 32 : 1, SUB = WIDE ? 32 : G;
    // published pivot rows, alternating by step: the columns, then 1/pivot and b
    __shared__ __align__(16) float2 rows[PER][2][NP + 2];
    __shared__ unsigned red[2][2][W];                       // WIDE: the warps' pivot candidates
    const int g = WIDE ? 0 : threadIdx.x / G, r = threadIdx.x % G;
    const long long sys0 = (long long)blockIdx.x * PER + g;
    const long long sys = sys0 < batch ? sys0 : batch - 1;   // spare groups repeat the last system
    const float2 *As = Ag + (size_t)sys * N * N;
    float2 a[NP];
#pragma unroll
    for (int c = 0; c < NP; ++c) a[c] = (r < N && c < N) ? As[r + (size_t)c * N] : make_float2(0.f, 0.f);
    float2 b = r < N ? bg[(size_t)sys * N + r] : make_float2(0.f, 0.f);
    float2 ipiv = make_float2(0.f, 0.f);
    unsigned pos = r;   // the row's place after the exchanges so far; rows >= N never take part
    auto barrier = [&]() {
        if (WIDE) __syncthreads();
        else __syncwarp();
    };
    fused::static_for<0, NP>([&](auto ic) __attribute__((always_inline)) {
        constexpr int i = decltype(ic)::value;
        if (i >= N) return;
        // the pivot: largest |a_ri|^2 of the rows left, the first of them; a NaN
        // is never larger, so it ranks below zero
        const bool left = (int)pos >= i && r < N;
        const float v = cabs2(a[i]);
        const unsigned key = left ? (v >= 0.f ? __float_as_uint(v) + 2u : 1u) : 0u;
        unsigned most = group_max<SUB>(key);
        unsigned first = group_min<SUB>(key == most ? pos : 0xffffu);
        if (WIDE) {
            if ((threadIdx.x & 31) == 0) {
                red[i & 1][0][threadIdx.x >> 5] = most;
                red[i & 1][1][threadIdx.x >> 5] = first;
            }
            __syncthreads();
            most = red[i & 1][0][0];
            first = red[i & 1][1][0];
#pragma unroll
            for (int w = 1; w < W; ++w) {
                const unsigned m = red[i & 1][0][w], p = red[i & 1][1][w];
                if (m > most || (m == most && p < first)) {
                    most = m;
                    first = p;
                }
            }
        }
        // rows without a comparable entry keep their order
        if (most <= 1u) first = i;
        const bool mine = left && pos == first;
        if (left && !mine && (int)pos == i) pos = first;
        float2 *row = rows[g][i & 1];
        // the columns right of the pivot, two a word from the first even one
        constexpr int c0 = (i + 1) & ~1;
        if (mine) {
            pos = i;
            // two quotients: the reciprocal of |p|^2 overflows below |p| = 5.4e-20, where
            // conj(p) / |p|^2 is still a number, and rounds once more (covariances and
            // solve of 16 k pixels at N = 32: 350 us by the reciprocal, 364 us so)
            const float pd = cabs2(a[i]);
            ipiv = make_float2(a[i].x / pd, -a[i].y / pd);
            *(float4 *)(row + NP) = make_float4(ipiv.x, ipiv.y, b.x, b.y);
#pragma unroll
            for (int c = c0; c < NP; c += 2) *(float4 *)(row + c) = make_float4(a[c].x, a[c].y, a[c + 1].x, a[c + 1].y);
        }
        barrier();
        // the buffer of step i is written again at step i+2, past the barrier of i+1
        if ((int)pos > i && r < N) {
            const float4 h = *(const float4 *)(row + NP);
            const float2 f = cmul(a[i], make_float2(h.x, h.y));
            const float2 nf = make_float2(-f.x, -f.y);
#pragma unroll
            for (int c = c0; c < NP; c += 2) {
                const float4 u = *(const float4 *)(row + c);   // columns past N are never used
                if (c > i) a[c] = cmac4(a[c], nf, make_float2(u.x, u.y));
                a[c + 1] = cmac4(a[c + 1], nf, make_float2(u.z, u.w));
            }
            b = cmac4(b, nf, make_float2(h.z, h.w));
        }
    });
    // back substitution; x_i from the row at place i
    float2 x = make_float2(0.f, 0.f);   // unknown of place r
    barrier();
    fused::static_for<0, NP>([&](auto ic) __attribute__((always_inline)) {
        constexpr int i = NP - 1 - decltype(ic)::value;
        if (i >= N) return;
        float2 *xs = rows[g][i & 1];
        if ((int)pos == i && r < N) *xs = cmul(b, ipiv);
        barrier();
        const float2 xi = *xs;
        if (r == i) x = xi;
        if ((int)pos < i) b = csub(b, cmul(a[i], xi));
    });
    if (sys0 < batch && r < N) xg[(size_t)sys * N + r] = x;
}

template <int NP, int G, int THREADS>
int launch(float2 *x, const float2 *A, const float2 *b, int N, long long batch, cudaStream_t s)
{
    const long long per = THREADS / G, blocks = (batch + per - 1) / per;
    lu_solve_kernel<NP, G, THREADS><<<(unsigned)blocks, THREADS, 0, s>>>(N, batch, A, b, x);
    return cudaGetLastError();
}

}  // namespace

int launch_lu_solve(float2 *x, const float2 *A, const float2 *b, int N, int batch, cudaStream_t s)
{
    // the columns held are the next of these sizes: a shorter row costs idle
    // columns in the update only up to there (8192 systems of N = 34: 339 us with 48
    // columns, 226 us with 36; two rows a lane of one warp 296 us, in shared memory as
    // before 348 us)
    if (N <= 8) return launch<8, 8, 128>(x, A, b, N, batch, s);
    if (N <= 16) return launch<16, 16, 128>(x, A, b, N, batch, s);
    if (N <= 24) return launch<24, 32, 128>(x, A, b, N, batch, s);
    if (N <= 32) return launch<32, 32, 128>(x, A, b, N, batch, s);
    if (N <= 36) return launch<36, 64, 64>(x, A, b, N, batch, s);
    if (N <= 40) return launch<40, 64, 64>(x, A, b, N, batch, s);
    if (N <= 48) return launch<48, 64, 64>(x, A, b, N, batch, s);
    if (N <= 64) return launch<64, 64, 64>(x, A, b, N, batch, s);
    return launch<72, 96, 96>(x, A, b, N, batch, s);
}

}  // namespace cgb
