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

// A warp takes 32 consecutive range pixels of one beam, a pixel per lane.  The
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
// hydrophones, bound by the line rate of L1; 158 us so, bound by
// issue, about 110 instructions an element).  Persistent CTAs, four an SM: the origin and
// the hydrophones' terms, as much FP64 as a run of pixels itself, are formed once
// a CTA (a CTA per 256 pixels: 164 us; three an SM at 75 registers 162 us,
// five 193 us).  The cube's rows run over
// the hydrophones, so the samples of 16 of them pass through shared memory and
// leave as whole 128-byte rows.
__global__ void __launch_bounds__(32 * kTdibWarps, 4) tdib_kernel(TdibDev t)
{
    __shared__ float2 hyd[kTdibMaxHydros];                       // (x_n, c_n)
    __shared__ float2 tile[kTdibWarps][32][kTdibChunk + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // origin: half the mean receiver position and depth (the same
    // lane-strided sums and butterfly in every warp)
    double sx = 0.0, sz = 0.0;
    for (int n = lane; n < t.n_hydros; n += 32) {
        sx += t.x_r[n];
        sz += t.D[n];
    }
    for (int o = 16; o; o >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, o);
        sz += __shfl_xor_sync(0xffffffffu, sz, o);
    }
    const double xx = 0.5 * sx / (double)t.n_hydros, zz = 0.5 * sz / (double)t.n_hydros;
    const float ku = t.ku, kc = t.kc;
    // |d| is at most a receiver's distance from the origin: whether d/(c dt) of
    // all of them stays below 2^21 samples (the FP32 floor below)
    bool far = false;
    for (int n = threadIdx.x; n < t.n_hydros; n += blockDim.x) {
        const double x = t.x_r[n], dd = t.D[n];
        hyd[n] = make_float2((float)x, (float)(x * x + dd * (dd - 2.0 * zz)));
        far |= !((fabs(x) + fabs(dd) + fabs(zz)) * ku < 2097152.0);
    }
    far = __syncthreads_or(far) || t.n_samples > (1 << 29);
    const int runs = (t.n_y + 31) / 32;
#pragma unroll 1
    for (long long wid = (long long)blockIdx.x * kTdibWarps + warp; wid < (long long)t.n_x * runs;
         wid += (long long)gridDim.x * kTdibWarps) {
        const int nx = (int)(wid / runs), y0 = (int)(wid % runs) * 32, np = min(32, t.n_y - y0);
        const int yl = y0 + min(lane, np - 1);   // lanes past the beam's end repeat its last pixel
        float a, r, r2, fr, bc;
        int b;
        {
            const double X = t.xarr[(size_t)nx * t.n_y + yl], Y = t.yarr[(size_t)nx * t.n_y + yl];
            const double ax = xx + X, rt2 = ax * ax + Y * Y + zz * zz, rt = sqrt(rt2);
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
        const int near = max(min(b, 1 << 30), -(1 << 30));   // no nearer to the axis than b
        const float qnan = __int_as_float(0x7fc00000);
        float2 acc[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = make_float2(0.f, 0.f);
        auto pass = [&](auto far_c) __attribute__((always_inline)) {
            constexpr bool FAR = decltype(far_c)::value;
            for (int n0 = 0; n0 < t.n_hydros; n0 += kTdibChunk) {
                const int nc = min(kTdibChunk, t.n_hydros - n0);
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
                if (t.Xd) {
                    // two rows of 16 hydrophones a store
                    const int col = lane % kTdibChunk;
                    float2 *o = t.Xd + ((size_t)nx * t.n_y + y0) * t.n_hydros + n0 + col;
        #pragma unroll 4
                    for (int p = lane / kTdibChunk; p < np; p += 32 / kTdibChunk)
                        if (col < nc) o[(size_t)p * t.n_hydros] = tile[warp][p][col];
                }
                __syncwarp();
            }
        };
        if (far) pass(std::true_type{});
        else pass(std::false_type{});
        if (t.image && lane < np) {
            const float2 s = cadd(cadd(acc[0], acc[1]), cadd(acc[2], acc[3]));
            t.image[(size_t)(y0 + lane) * t.n_x + nx] = cscale(s, 1.0f / (float)t.n_hydros);
        }
    }
}

int launch_tdib(const TdibDev &t, cudaStream_t s)
{
    if (t.n_hydros > kTdibMaxHydros) return cudaErrorNotSupported;
    const long long warps = (long long)t.n_x * ((t.n_y + 31) / 32);
    const long long blocks = (warps + kTdibWarps - 1) / kTdibWarps;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
        (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tdib_kernel, 32 * kTdibWarps, 0)) != cudaSuccess)
        return e;
    const long long resident = (long long)sms * per_sm;
    tdib_kernel<<<(unsigned)(blocks < resident ? blocks : resident), 32 * kTdibWarps, 0, s>>>(t);
    return cudaGetLastError();
}

}  // namespace cgb
