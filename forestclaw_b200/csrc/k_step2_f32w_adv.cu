// k_step2_f32w_adv.cu -- FP32-wave instantiations (built with --use_fast_math; FP64 accumulation)
// of the fused update for scalar advection (plane and manifold; k_adv.cuh): per patch size
// the variants with the MC limiter fixed at compile time, then those for any method.
#include "k_adv.cuh"
#include "fc2d_b200.h"

namespace fcb {

const Step2Variant* step2_table_f32w_adv(int* n)
{
    static const Step2Variant table[] = {
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION, AdvPlane, 32, 448, 2, float, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION, AdvPlane, 32, 672, 2, float, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION, AdvPlane, 32, 448, 2, float, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION, AdvPlane, 32, 672, 2, float, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION, AdvPlane, 16, 416, 2, float, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION, AdvPlane, 16, 416, 4, float, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION, AdvPlane, 16, 224, 4, float, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION, AdvPlane, 16, 416, 2, float, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION, AdvPlane, 16, 224, 4, float, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 32, 448, 2, float, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 32, 672, 2, float, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 32, 448, 2, float, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 32, 672, 2, float, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 16, 416, 2, float, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 16, 416, 3, float, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 16, 224, 4, float, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 16, 416, 2, float, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 16, 224, 4, float, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 8, 160, 4, float, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 8, 160, 8, float, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP32WAVE, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 8, 160, 4, float, 0),
    };
    *n = (int)(sizeof(table) / sizeof(table[0]));
    return table;
}

}  // namespace fcb
