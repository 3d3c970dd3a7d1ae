// Fused element-space kernel instantiations for L = 16, temporal window T = 3.
// The autotuner in capon_api.cu picks one per (L, K, M) shape; a candidate
// compiled for a fixed M reports cudaErrorNotSupported for other M.
#include "capon_fused.cuh"

namespace cgb {
int fused_l16r_launch(const FramesParam &fp, int mode, unsigned *st, int n, cudaStream_t s);
size_t fused_l16r_smem(int K, int M);
size_t fused_l16r_stash(int num_sms);

namespace {
int launch_0(const FramesParam &fp, int mode, unsigned *st, int n, cudaStream_t s)
{
    return fused::launch_any<fused::Cfg<16, 4, 8, 1, 3, 0, true>>(fp, mode, st, n, s);
}

// three CTAs of four warps an SM: at 168 registers a thread instead of 255 the
// L = 16 triangle still fits, and half as many warps again cover each other's
// waits (where shared memory leaves room for them).  K = 1: [256][1024][32], z and
// P, 0.261 -> 0.236 ms; [61][507][37] with weights 57 -> 45 us
int launch_1(const FramesParam &fp, int mode, unsigned *st, int n, cudaStream_t s)
{
    return fused::launch_any<fused::Cfg<16, 4, 4, 1, 3, 0, false, false, 3>>(fp, mode, st, n, s);
}
int launch_2(const FramesParam &fp, int mode, unsigned *st, int n, cudaStream_t s)
{
    return fused::launch_any<fused::Cfg<16, 4, 4, 1, 3, 32, false, false, 3>>(fp, mode, st, n, s);
}
// the same with one row stride for every M <= 40: K = 2, [200][507][30], z and P,
// 0.175 -> 0.115 ms
int launch_3(const FramesParam &fp, int mode, unsigned *st, int n, cudaStream_t s)
{
    return fused::launch_any<fused::Cfg<16, 4, 4, 1, 3, 0, false, false, 3, 42>>(fp, mode, st, n, s);
}

const FusedCandidate kCand[] = {
    {"L16.G4.W4.N1.B3.M32.T3", 16, 3, 32, launch_2,
     fused::smem_bytes<fused::Cfg<16, 4, 4, 1, 3, 32, false, false, 3>>},
    {"L16.G4.W4.N1.B3.X42.T3", 16, 3, 0, launch_3,
     fused::smem_bytes<fused::Cfg<16, 4, 4, 1, 3, 0, false, false, 3, 42>>},
    {"L16.G4.W4.N1.B3.T3", 16, 3, 0, launch_1, fused::smem_bytes<fused::Cfg<16, 4, 4, 1, 3, 0, false, false, 3>>},
    {"L16.G4.W8.N1.sync.T3", 16, 3, 0, launch_0, fused::smem_bytes<fused::Cfg<16, 4, 8, 1, 3, 0, true>>},
    // the refinement modes (capon_fused_l16r.cu)
    {"L16.G8.W8.refine", 16, 0, 0, fused_l16r_launch, fused_l16r_smem, fused_l16r_stash, true},
};
}  // namespace

int fused_candidates_l16_t3(const FusedCandidate **out)
{
    *out = kCand;
    return (int)(sizeof(kCand) / sizeof(kCand[0]));
}

}  // namespace cgb
