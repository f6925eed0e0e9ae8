// k_step2_f64_sw.cu -- FP64 instantiations (built with -fmad=false: bitwise equal to the FP64 CPU path)
// of the fused update for shallow water (Roe and f-wave): per patch size the variants with the MC limiter
// fixed at compile time (k_wave.cuh), then those for any method.
#include "k_wave.cuh"
#include "fc2d_b200.h"

namespace fcb {

const Step2Variant* step2_table_f64_sw(int* n)
{
    static const Step2Variant table[] = {
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 16, 384, 2, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 16, 352, 2, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 16, 352, 1, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 16, 384, 2, double, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 16, 352, 2, double, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 8, 128, 6, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 8, 128, 5, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 8, 128, 4, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 8, 128, 6, double, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 8, 128, 4, double, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 16, 384, 2, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 16, 352, 2, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 16, 352, 1, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 16, 384, 2, double, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 16, 352, 2, double, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 8, 128, 6, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 8, 128, 5, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 8, 128, 4, double, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 8, 128, 6, double, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 8, 128, 4, double, 0),
    };
    *n = (int)(sizeof(table) / sizeof(table[0]));
    return table;
}

}  // namespace fcb
