// k_step2_f32w_sw.cu -- FP32-wave instantiations (built with --use_fast_math; FP64 accumulation)
// of the fused update for shallow water (Roe and f-wave): per patch size the variants with the MC limiter
// fixed at compile time (k_wave.cuh), then those for any method.
#include "k_wave.cuh"
#include "fc2d_b200.h"

namespace fcb {

const Step2Variant* step2_table_f32w_sw(int* n)
{
    static const Step2Variant table[] = {
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 16, 384, 3, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 16, 352, 3, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 16, 384, 2, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 16, 384, 3, float, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 16, 384, 2, float, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 8, 128, 8, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 8, 128, 6, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 8, 128, 4, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 8, 128, 8, float, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_ROE, WaveShallowRoe, 8, 128, 6, float, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 16, 384, 3, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 16, 352, 3, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 16, 384, 2, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 16, 384, 3, float, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 16, 384, 2, float, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 8, 128, 8, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 8, 128, 6, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 8, 128, 4, float, 4),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 8, 128, 8, float, 0),
        FCB_WAVE_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_SW_FWAVE, WaveShallowFWave, 8, 128, 6, float, 0),
    };
    *n = (int)(sizeof(table) / sizeof(table[0]));
    return table;
}

}  // namespace fcb
