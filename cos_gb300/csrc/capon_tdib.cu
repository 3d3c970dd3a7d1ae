// Time-domain steering (TDIB) for sm_103a: the step before the Capon path.
//
// Follows framework/beamformer/delay/tdibC.pyx:9-67: for beam nx, range pixel
// y and hydrophone n, with the transmitter/receiver origin at
// (xx, zz) = (mean(x_r)/2, mean(D)/2),
//     r_t   = sqrt((xx + X)^2 + Y^2 + zz^2)
//     r_r   = sqrt((xx + X - x_r[n])^2 + Y^2 + (zz - D[n])^2)
//     tau   = (r_t + r_r) / c
//     Xd    = interp_linear(mfdata[n], tau) * exp(j 2 pi fc tau)
// (NaN outside the time axis, as scipy's interp1d with bounds_error=False),
// and the delay-and-sum image is the mean of Xd over hydrophones.  The
// steered cube Xd[nx][y][n] is the Capon path's input layout.
//
// The carrier needs the delay to ~1e-9 relative, beyond FP32; GB300's FP64
// rate is a small fraction of its FP32 rate.  So FP64 is spent once per pixel
// (the base delay and phase) and the per-hydrophone terms are FP32 corrections
// of a few samples / cycles (see tdib_kernel).  Measured against the FP64
// restatement: ~2e-6 of the cube's scale.
#include <type_traits>

#include "capon_common.cuh"
#include "capon_internal.h"
#include "../../include/cos_capon.h"

namespace cgb {

static constexpr int kTdibMaxHydros = 256;
static constexpr int kTdibWarps = 8;
// hydrophones per transposed tile: 32 pixels x 16 complex, 4.4 KB a warp
static constexpr int kTdibChunk = 16;

// a >= 0 to about half an ulp and q = n / d to about an ulp: the unit's
// approximation and one residual step (Heron's, and the quotient's own remainder)
COS_DEV float root_of(float a)
{
    a = fmaxf(a, 1e-30f);
    const float y = rsqrtf(a), s = a * y;
    return fmaf(0.5f * y, fmaf(-s, s, a), s);
}
COS_DEV float quotient(float n, float d)
{
    const float y = __fdividef(1.f, d), q = n * y;
    return fmaf(y, fmaf(-q, d, n), q);
}

// A warp takes 32 consecutive pixels of the fan, beam after beam, a pixel per lane.  The
// lane evaluates the FP64 part of its pixel once: r_t, the base delay 2 r_t / c
// split into an integer sample index and a fraction, and the base carrier phase
// fc 2 r_t / c reduced to a fraction of a cycle.  Per hydrophone only the small
// difference d = r_r - r_t is needed; it is formed in FP32 without cancellation,
//     e = r_r^2 - r_t^2 = c_n - 2 ax x_n,   c_n = x_n^2 + D_n^2 - 2 zz D_n
//     d = e / (r_t + sqrt(r_t^2 + e)),
// and enters the sample index as d/(c dt) and the phase as fc d/c (a few
// samples / cycles, so FP32 keeps ~1e-6 of a cycle).
//
// The pixel sits on the lane, not the hydrophone, for the gathers: neighbouring
// range pixels read neighbouring samples of one channel, a few cache lines a
// load, where 32 channels are 32 lines (263 us for [256][2048] pixels x 64
// hydrophones, bound by the line rate of L1; 152 us so, bound by
// issue, about 110 instructions an element).  Persistent CTAs, four an SM: the origin and
// the hydrophones' terms are formed once a CTA, the origin by one of its warps (by all
// of them: 159 us).  (A CTA per 256 pixels is 4 % slower, three an SM at 75 registers 3 %,
// five 22 %.)  The cube's rows run over
// the hydrophones, so the samples of 16 of them pass through shared memory and
// leave as whole 128-byte rows.
//
// SPLIT, for calls that leave warps idle: `parts` warps of a CTA share 32 pixels, cw
// hydrophones (4, 8 or 16) each in turn; the FP64 part is the first one's, and their
// image sums meet in shared memory.  [8][1] pixels x 250 hydrophones: 25 us, 69 us by
// one warp (26 us with a hydrophone per lane); [512][2] x 64: 18 us, 32 us (23 us).
template <bool SPLIT>
__global__ void __launch_bounds__(32 * kTdibWarps, 4) tdib_kernel(TdibDev t, int parts, int cw)
{
    if (!SPLIT) {
        parts = 1;
        cw = kTdibChunk;
    }
    __shared__ float2 hyd[kTdibMaxHydros];                       // (x_n, c_n)
    __shared__ double origin[2];
    __shared__ float base[SPLIT ? kTdibWarps : 1][6][32];        // a group's FP64 results
    __shared__ float2 part[SPLIT ? kTdibWarps : 1][32];          // image sums of the warps
    __shared__ float2 tile[kTdibWarps][32][kTdibChunk + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // origin: half the mean receiver position and depth, by one warp (FP64 of all
    // eight would take as long as a run of pixels)
    if (warp == 0) {
        double sx = 0.0, sz = 0.0;
        for (int n = lane; n < t.n_hydros; n += 32) {
            sx += t.x_r[n];
            sz += t.D[n];
        }
        for (int o = 16; o; o >>= 1) {
            sx += __shfl_xor_sync(0xffffffffu, sx, o);
            sz += __shfl_xor_sync(0xffffffffu, sz, o);
        }
        if (lane == 0) {
            origin[0] = 0.5 * sx / (double)t.n_hydros;
            origin[1] = 0.5 * sz / (double)t.n_hydros;
        }
    }
    __syncthreads();
    const float ku = t.ku, kc = t.kc;
    // |d| is at most a receiver's distance from the origin: whether d/(c dt) of
    // all of them stays below 2^21 samples (the FP32 floor below)
    bool far = false;
    for (int n = threadIdx.x; n < t.n_hydros; n += blockDim.x) {
        const double x = t.x_r[n], dd = t.D[n], zz = origin[1];
        hyd[n] = make_float2((float)x, (float)(x * x + dd * (dd - 2.0 * zz)));
        far |= !((fabs(x) + fabs(dd) + fabs(zz)) * ku < 2097152.0);
    }
    far = __syncthreads_or(far) || t.n_samples > (1 << 29);
    const long long pixels = (long long)t.n_x * t.n_y;
    const unsigned runs = (unsigned)((pixels + 31) / 32);
    const int groups = SPLIT ? kTdibWarps / parts : kTdibWarps, group = warp / parts, sub = SPLIT ? warp % parts : 0;
#pragma unroll 1
    for (unsigned u = blockIdx.x * groups; u < runs; u += gridDim.x * groups) {
        // a group past the end leaves, or, where its CTA's warps meet, repeats the last
        // run and stores nothing
        if (!SPLIT && u + group >= runs) break;
        const long long g0 = (long long)min(u + group, runs - 1) * 32;
        float a, r, r2, fr, bc;
        int b;
        if (sub == 0) {
            const long long gl = min(g0 + lane, pixels - 1);   // lanes past the end repeat the last pixel
            const double X = t.xarr[gl], Y = t.yarr[gl], zz = origin[1];
            const double ax = origin[0] + X, rt2 = ax * ax + Y * Y + zz * zz, rt = sqrt(rt2);
            const double tau0 = 2.0 * rt * t.inv_c;
            // a quotient: a delay on the last sample must not come out past it
            const double u0 = (tau0 - t.t0) / t.dt;
            const double fu = floor(u0);
            const double cyc = t.fc * tau0;
            b = (int)fu;
            fr = (float)(u0 - fu);
            bc = (float)(cyc - floor(cyc));
            a = (float)ax;
            r = (float)rt;
            r2 = (float)rt2;
        }
        if (SPLIT) {
            // the group's other warps take them from the first
            float(*const v)[32] = base[group];
            if (sub == 0) {
                v[0][lane] = a;
                v[1][lane] = r;
                v[2][lane] = r2;
                v[3][lane] = fr;
                v[4][lane] = bc;
                v[5][lane] = __int_as_float(b);
            }
            __syncthreads();
            a = v[0][lane];
            r = v[1][lane];
            r2 = v[2][lane];
            fr = v[3][lane];
            bc = v[4][lane];
            b = __float_as_int(v[5][lane]);
        }
        const int near = max(min(b, 1 << 30), -(1 << 30));   // no nearer to the axis than b
        const float qnan = __int_as_float(0x7fc00000);
        float2 acc[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = make_float2(0.f, 0.f);
        auto pass = [&](auto far_c) __attribute__((always_inline)) {
            constexpr bool FAR = decltype(far_c)::value;
            for (int n0 = sub * cw; n0 < t.n_hydros; n0 += parts * cw) {
                const int nc = min(cw, t.n_hydros - n0);
                // four hydrophones at a time: their gathers in flight together
                for (int k0 = 0; k0 < nc; k0 += 4) {
                    float2 lo[4], hi[4];
                    float wgt[4], ph[4];
                    bool out[4];
        #pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int n = min(n0 + k0 + q, t.n_hydros - 1);
                        const float2 h = hyd[n];
                        const float e = h.y - 2.f * a * h.x;
                        const float d = quotient(e, r + root_of(r2 + e));
                        const float uf = fr + d * ku;
                        // floor(uf): adding 1.5 2^23 leaves the nearest integer in the
                        // low bits (|uf| < 2^22), all on the FP32 pipe
                        float fl;
                        int i;
                        bool in, last;   // on the time axis; at its last sample
                        if (FAR) {
                            fl = floorf(uf);
                            const long long il = (long long)b + (long long)fl;   // b saturates for far-away delays
                            last = il == t.n_samples - 1;
                            in = il >= 0 && (il < t.n_samples - 1 || (last && uf <= fl));
                            i = in ? (int)il : 0;
                        } else {
                            fl = (uf + 12582912.f) - 12582912.f;
                            fl -= fl > uf ? 1.f : 0.f;
                            i = near + (__float_as_int(fl + 12582912.f) - 0x4b400000);
                            last = i == t.n_samples - 1;
                            in = (unsigned)i < (unsigned)(t.n_samples - 1) || (last && uf <= fl);
                            i = in ? i : 0;
                        }
                        out[q] = !in;
                        const float2 *row = t.mf + (size_t)n * t.n_samples + i;
                        lo[q] = row[0];
                        hi[q] = row[in && last ? 0 : 1];
                        wgt[q] = uf - fl;
                        ph[q] = bc + d * kc;   // sincospi reduces it exactly
                    }
        #pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float2 sm = make_float2(lo[q].x + wgt[q] * (hi[q].x - lo[q].x),
                                                      lo[q].y + wgt[q] * (hi[q].y - lo[q].y));
                        float sn, cs;
                        sincospif(2.0f * ph[q], &sn, &cs);
                        float2 v = cmul(sm, make_float2(cs, sn));
                        if (out[q]) v = make_float2(qnan, qnan);
                        if (k0 + q < nc) {
                            tile[warp][lane][k0 + q] = v;
                            acc[q] = cadd(acc[q], v);
                        }
                    }
                }
                __syncwarp();
                const int np = u + group < runs ? (int)min(32LL, pixels - g0) : 0;
                if (t.Xd) {
                    // two rows of 16 hydrophones a store
                    const int col = lane & (cw - 1);
                    float2 *o = t.Xd + (size_t)g0 * t.n_hydros + n0 + col;
        #pragma unroll 4
                    for (int p = lane / cw; p < np; p += 32 / cw)
                        if (col < nc) o[(size_t)p * t.n_hydros] = tile[warp][p][col];
                }
                __syncwarp();
            }
        };
        if (far) pass(std::true_type{});
        else pass(std::false_type{});
        if (t.image) {
            float2 v = cadd(cadd(acc[0], acc[1]), cadd(acc[2], acc[3]));
            if (SPLIT) {
                part[warp][lane] = v;
                __syncthreads();
                if (sub == 0)
                    for (int q = 1; q < parts; ++q) v = cadd(v, part[warp + q][lane]);
            }
            if (sub == 0 && u + group < runs && g0 + lane < pixels) {
                const long long nx = (g0 + lane) / t.n_y, y = g0 + lane - nx * t.n_y;
                t.image[(size_t)y * t.n_x + nx] = cscale(v, 1.0f / (float)t.n_hydros);
            }
        }
        if (SPLIT) __syncthreads();   // the readers of base and part are done
    }
}

int launch_tdib(const TdibDev &t, cudaStream_t s)
{
    if (t.n_hydros > kTdibMaxHydros) return cudaErrorNotSupported;
    const long long runs = ((long long)t.n_x * t.n_y + 31) / 32;
    if (runs > 0x7fffffffLL) return cudaErrorInvalidValue;   // 2^36 pixels: 1 TB of coordinates
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
        (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tdib_kernel<false>, 32 * kTdibWarps, 0)) !=
            cudaSuccess)
        return e;
    const long long resident = (long long)sms * per_sm;
    // few pixels: a warp's time is that of its hydrophones, one batch of four after
    // the other, so as many warps as would be idle share them
    int parts = 1;
    while (parts < kTdibWarps && runs * parts * 2 <= resident * kTdibWarps && parts * 4 < t.n_hydros) parts *= 2;
    const int each = (t.n_hydros + parts - 1) / parts, cw = each <= 4 ? 4 : each <= 8 ? 8 : kTdibChunk;
    const long long groups = kTdibWarps / parts, blocks = (runs + groups - 1) / groups;
    const unsigned grid = (unsigned)(blocks < resident ? blocks : resident);
    if (parts > 1)
        tdib_kernel<true><<<grid, 32 * kTdibWarps, 0, s>>>(t, parts, cw);
    else
        tdib_kernel<false><<<grid, 32 * kTdibWarps, 0, s>>>(t, 1, kTdibChunk);
    return cudaGetLastError();
}

}  // namespace cgb
