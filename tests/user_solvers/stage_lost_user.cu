// The package's update kernels told that their staging copies never arrive (FCB_STAGE_LOST; the
// copies do arrive and are waited for), registered as application solvers.
#define FCB_STAGE_LOST
#include "fc2d_b200_user.cuh"
#include "k_adv.cuh"
#include "k_wave.cuh"

using namespace fcb;

// occupancy targets that the package does not instantiate, so that these are kernels of their own
extern "C" int stage_lost_register_inline(fc2d_b200_solver_t* s)
{
    static const Step2Variant table[] = {
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_USER, WaveShallowRoe, 8, 128, 1, double, 0)};
    return fc2d_b200_set_user_variants(s, table, 1, FC2D_B200_USER_ABI, 3, 3, 0);
}
extern "C" int stage_lost_register_advection(fc2d_b200_solver_t* s)
{
    static const Step2Variant table[] = {
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_USER, AdvPlane, 8, 160, 1, double, 0)};
    return fc2d_b200_set_user_variants(s, table, 1, FC2D_B200_USER_ABI, 1, 1, 2);
}
