// k_step2_f32w_euler.cu -- FP32-wave instantiations (built with --use_fast_math; FP64 accumulation)
// of the fused update for the exact Euler solver (k_wave.cuh): MC limiter fixed at compile time, then any method.
#include "k_wave.cuh"
#include "fc2d_b200.h"

namespace fcb {

const Step2Variant* step2_table_f32w_euler(int* n)
{
    static const Step2Variant table[] = {
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 16, 384, 2, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 16, 352, 2, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 16, 352, 1, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 16, 384, 2, float, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 16, 352, 2, float, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 8, 128, 6, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 8, 128, 5, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 8, 128, 4, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 8, 128, 6, float, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_EULER_EXACT, WaveEulerExact, 8, 128, 4, float, 0),
    };
    *n = (int)(sizeof(table) / sizeof(table[0]));
    return table;
}

}  // namespace fcb
