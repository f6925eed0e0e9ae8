// k_step2_f64_euler.cu -- FP64 instantiations (built with -fmad=false: bitwise equal to the FP64 CPU path)
// of the fused update for the exact Euler solver (k_wave.cuh): MC limiter fixed at compile time, then any method.
#include "k_wave.cuh"
#include "fc2d_b200.h"

namespace fcb {

const Step2Variant* step2_table_f64_euler(int* n)
{
    static const Step2Variant table[] = {
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 16, 384, 1, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 16, 352, 1, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 16, 384, 1, double, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 8, 128, 4, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 8, 128, 3, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 8, 128, 2, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 8, 128, 4, double, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 8, 128, 3, double, 0),
    };
    *n = (int)(sizeof(table) / sizeof(table[0]));
    return table;
}

}  // namespace fcb
