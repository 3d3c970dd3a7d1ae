// Solve stage of the general element-space path: L <= 64, z and P.
#include "capon_general.cuh"

namespace cgb {
int general_solve_l64_zp(const FrameDev &f, const float2 *work, unsigned *status, int num_sms, cudaStream_t s)
{
    return general::launch_solve<general::SolveCfg<64, 32, 16, 8, 1>, false>(f, work, status, num_sms, s);
}
}  // namespace cgb
