// Fused element-space kernel, L = 48, any T, 12 warps x 2 pixels, any M: the z/P, w and R modes (the
// blocked per-pixel path of capon_fused_wide.cuh); the candidate table is in
// capon_fused_l48.cu.
#include "capon_fused.cuh"

namespace cgb {
using CL48B = fused::Cfg<48, 16, 12, 1, 0, 0, false>;
int fused_l48b_launch(const FramesParam &fp, int mode, unsigned *st, int n, cudaStream_t s)
{
    return fused::launch_basic<CL48B>(fp, mode, st, n, s);
}
size_t fused_l48b_smem(int K, int M) { return fused::smem_bytes<CL48B>(K, M); }
}  // namespace cgb
