// k_step2_f64_adv.cu -- FP64 instantiations (built with -fmad=false: bitwise equal to the FP64 CPU path)
// of the fused update for scalar advection (plane and manifold; k_adv.cuh): per patch size
// the variants with the MC limiter fixed at compile time, then those for any method.
#include "k_adv.cuh"
#include "fc2d_b200.h"

namespace fcb {

const Step2Variant* step2_table_f64_adv(int* n)
{
    static const Step2Variant table[] = {
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION, AdvPlane, 32, 448, 2, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION, AdvPlane, 32, 672, 2, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION, AdvPlane, 32, 448, 2, double, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION, AdvPlane, 32, 672, 2, double, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION, AdvPlane, 16, 416, 2, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION, AdvPlane, 16, 416, 4, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION, AdvPlane, 16, 224, 4, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION, AdvPlane, 16, 416, 2, double, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION, AdvPlane, 16, 224, 4, double, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION, AdvPlane, 8, 160, 4, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION, AdvPlane, 8, 160, 8, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION, AdvPlane, 8, 160, 4, double, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 32, 448, 2, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 32, 672, 2, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 32, 448, 2, double, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 32, 672, 2, double, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 16, 416, 2, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 16, 416, 3, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 16, 224, 4, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 16, 416, 2, double, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 16, 224, 4, double, 0),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 8, 160, 4, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 8, 160, 8, double, 4),
        FCB_ADV_VARIANT(FC2D_B200_PREC_FP64, FC2D_B200_RP_ADVECTION_MANIFOLD, AdvManifold, 8, 160, 4, double, 0),
    };
    *n = (int)(sizeof(table) / sizeof(table[0]));
    return table;
}

}  // namespace fcb
