// Low-complexity adaptive (LCA) window selection for sm_103a.
//
// Follows framework/beamformer/lca/lcac.py (Z[Ny][Nx][Nw], the layout whose
// indexing is consistent; lcacx.pyx:175-216 is the same algorithm):
//   * wrf of size 1 x 1 with a nonzero value: per pixel the window of least
//     |Z| (argmin over w), for every pixel;
//   * otherwise, for interior pixels y in [Ymid, Ny-Ymid), x in [Xmid, Nx-Xmid):
//       s_w = sum_{yy,xx} |Z[y+yy-Ymid][x+xx-Xmid][w]|^2 wrf[yy][xx],
//     the first w of least s_w is selected; img = Z[y][x][w*], win = w*;
//     border pixels keep img = 0, win = 0.
//
// One pass: a CTA brings its tile of Z, with the filter's halo, through |.|^2
// into shared memory, up to W = 4 or 8 windows a pixel at a time (more go in
// chunks, the best so far in registers), and a thread per pixel carries the W
// sums through the filter (FP32, yy then xx), a tap being one weight and one or
// two 16-byte loads for all W windows.  What bounds it: issue, about 15
// instructions a tap, then the read of Z; a [2048][256] image with 8 windows and a
// 5 x 1 filter takes 16 us (2.4 TB/s over Z once and the outputs; 18 us with two CTAs
// an SM instead of three).  As two passes
// over memory, the planes |Z|^2 in HBM between them, it took 60 us; with a scalar
// load, a multiply-add and the index arithmetic for every tap and window, 55 us.
#include <algorithm>
#include <type_traits>

#include "capon_common.cuh"
#include "capon_internal.h"
#include "../../include/cos_capon.h"

namespace cgb {

static constexpr int kLcaTX = 32, kLcaTY = 16, kLcaThreads = 512;

// W: windows a pixel holds in shared memory, S: its stride there in floats (8
// lanes of a 16-byte load fall on all 32 banks: 4 and 12)
template <int W>
__global__ void __launch_bounds__(kLcaThreads, 3) lca_kernel(LcaDev a)
{
    constexpr int S = W == 4 ? 4 : 12;
    extern __shared__ __align__(16) float pw[];
    const int x0 = blockIdx.x * kLcaTX, y0 = blockIdx.y * kLcaTY;
    const int cols = kLcaTX + a.Xf - 1, rows = kLcaTY + a.Yf - 1;
    const int tid = threadIdx.x, tx = tid % kLcaTX, ty = tid / kLcaTX, x = x0 + tx, y = y0 + ty;
    const bool in = x < a.Nx && y < a.Ny;
    // a 1 x 1 filter has no border: Ymid = Xmid = 0
    const bool inner = in && y >= a.Ymid && y < a.Ny - a.Ymid && x >= a.Xmid && x < a.Nx - a.Xmid;
    const float inv = 1.f / (float)cols;
    // a tile that the filter's border covers needs none of Z (an image of [16][16], 33
    // windows and a 255 x 1 filter: 67 -> 14 us)
    const bool none = max(a.Ymid, y0) >= min(a.Ny - a.Ymid, y0 + kLcaTY) ||
                      max(a.Xmid, x0) >= min(a.Nx - a.Xmid, x0 + kLcaTX);
    int best = 0;
    float bv = 0.f;
    // windows w0 .. w0+nw-1, at most 4 Q of them
    auto chunk = [&](const int w0, const int nw, auto qc) __attribute__((always_inline)) {
        constexpr int Q = decltype(qc)::value;
        if (w0) __syncthreads();  // the last chunk's readers are done
#pragma unroll 5
        for (int i = tid; i < rows * cols * (4 * Q); i += kLcaThreads) {
            const int px = i / (4 * Q), w = i % (4 * Q);
            const int r = small_div(px, inv);
            const int yy = y0 - a.Ymid + r, xx = x0 - a.Xmid + px - r * cols;
            float v = 0.f;
            if (w < nw && yy >= 0 && yy < a.Ny && xx >= 0 && xx < a.Nx)
                v = cabs2(a.Z[((long long)yy * a.Nx + xx) * a.Nw + (w0 + w)]);
            pw[px * S + w] = v;
        }
        __syncthreads();
        if (inner) {
            float s[4 * Q];
#pragma unroll
            for (int w = 0; w < 4 * Q; ++w) s[w] = 0.f;
            const float *p = pw + (ty * cols + tx) * S;
            if (a.single) {
#pragma unroll
                for (int w = 0; w < 4 * Q; ++w) s[w] = p[w];
            } else {
                for (int yy = 0, k = 0; yy < a.Yf; ++yy, p += (cols - a.Xf) * S)
#pragma unroll 1
                    for (int xx = 0; xx < a.Xf; ++xx, ++k, p += S) {
                        const float wgt = a.wrf[k];
#pragma unroll
                        for (int q = 0; q < Q; ++q) {
                            const float4 v = ((const float4 *)p)[q];
                            s[4 * q] = fmaf(v.x, wgt, s[4 * q]);
                            s[4 * q + 1] = fmaf(v.y, wgt, s[4 * q + 1]);
                            s[4 * q + 2] = fmaf(v.z, wgt, s[4 * q + 2]);
                            s[4 * q + 3] = fmaf(v.w, wgt, s[4 * q + 3]);
                        }
                    }
            }
#pragma unroll
            for (int w = 0; w < 4 * Q; ++w)
                if (w < nw && (w0 + w == 0 || s[w] < bv)) {
                    bv = s[w];
                    best = w0 + w;
                }
        }
    };
    for (int w0 = 0; w0 < a.Nw && !none; w0 += W) {
        const int nw = min(W, a.Nw - w0);
        if (W > 4 && nw <= 4) chunk(w0, nw, std::integral_constant<int, 1>{});   // the last of them
        else chunk(w0, nw, std::integral_constant<int, W / 4>{});
    }
    if (in) {
        const long long pix = (long long)y * a.Nx + x;
        a.img[pix] = inner ? a.Z[pix * a.Nw + best] : make_float2(0.f, 0.f);
        if (a.win) a.win[pix] = best;
    }
}

template <int W>
static int launch_w(const LcaDev &a, cudaStream_t s)
{
    const size_t smem = (size_t)(kLcaTX + a.Xf - 1) * (kLcaTY + a.Yf - 1) * (W == 4 ? 4 : 12) * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(lca_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)((a.Nx + kLcaTX - 1) / kLcaTX), (unsigned)((a.Ny + kLcaTY - 1) / kLcaTY));
    lca_kernel<W><<<grid, kLcaThreads, smem, s>>>(a);
    return cudaGetLastError();
}

int launch_lca(const LcaDev &a, cudaStream_t s)
{
    // W = 4 for few windows, and where the halo of a long filter (up to 256 taps)
    // leaves no room for 8: at most 32 x 271 pixels of 16 bytes, 139 KB
    const size_t n = (size_t)(kLcaTX + a.Xf - 1) * (kLcaTY + a.Yf - 1);
    return a.Nw <= 4 || n * 12 * sizeof(float) > 112 * 1024 ? launch_w<4>(a, s) : launch_w<8>(a, s);
}

}  // namespace cgb
