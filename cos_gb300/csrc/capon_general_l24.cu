// Solve stage of the general element-space path: L <= 8, 16 and 24.
#include "capon_general.cuh"

namespace cgb {
int general_solve_l8_zp(const FrameDev &f, const float2 *work, unsigned *status, int num_sms, cudaStream_t s)
{
    return general::launch_solve<general::SolveCfg<8, 4, 8, 8, 4>, false>(f, work, status, num_sms, s);
}
int general_solve_l8_w(const FrameDev &f, const float2 *work, unsigned *status, int num_sms, cudaStream_t s)
{
    return general::launch_solve<general::SolveCfg<8, 4, 8, 8, 4>, true>(f, work, status, num_sms, s);
}
int general_solve_l16_zp(const FrameDev &f, const float2 *work, unsigned *status, int num_sms, cudaStream_t s)
{
    return general::launch_solve<general::SolveCfg<16, 4, 8, 8, 2>, false>(f, work, status, num_sms, s);
}
int general_solve_l16_w(const FrameDev &f, const float2 *work, unsigned *status, int num_sms, cudaStream_t s)
{
    return general::launch_solve<general::SolveCfg<16, 4, 8, 8, 2>, true>(f, work, status, num_sms, s);
}
int general_solve_l24_zp(const FrameDev &f, const float2 *work, unsigned *status, int num_sms, cudaStream_t s)
{
    return general::launch_solve<general::SolveCfg<24, 8, 8, 6, 2>, false>(f, work, status, num_sms, s);
}
int general_solve_l24_w(const FrameDev &f, const float2 *work, unsigned *status, int num_sms, cudaStream_t s)
{
    return general::launch_solve<general::SolveCfg<24, 8, 8, 6, 2>, true>(f, work, status, num_sms, s);
}
}  // namespace cgb
