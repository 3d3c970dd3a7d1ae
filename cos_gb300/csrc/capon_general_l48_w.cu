// Solve stage of the general element-space path: L <= 48, with the weights.
#include "capon_general.cuh"

namespace cgb {
int general_solve_l48_w(const FrameDev &f, const float2 *work, unsigned *status, int num_sms, cudaStream_t s)
{
    return general::launch_solve<general::SolveCfg<48, 16, 16, 8, 1>, true>(f, work, status, num_sms, s);
}
}  // namespace cgb
