// The compiled shapes of the two-sweep 3D kernel: consumer warps, rows per warp,
// ring stages.
#include "j3d_pair.cuh"

#include "cfm.h"

namespace cfm {

namespace {

template <int CW, int RPW, int S>
long long tiles(int precision, int nx, int ny) {
    using D = J3PairGeom<double, CW, RPW, S>;
    using F = J3PairGeom<float, CW, RPW, S>;
    return precision == CFM_FP64 ? (long long)j3p_tiles_x<D>(nx) * j3p_tiles_y<D>(ny)
                                 : (long long)j3p_tiles_x<F>(nx) * j3p_tiles_y<F>(ny);
}

template <int CW, int RPW, int S, bool VEC>
J3PairShape make() {
    using D = J3PairGeom<double, CW, RPW, S>;
    using F = J3PairGeom<float, CW, RPW, S>;
    static_assert(D::SMEM == F::SMEM, "a lane holds 16 bytes per row in either precision");
    return {CW, RPW, S,
            {{(const void *)j3d_pair_kernel<double, CW, RPW, S, false, VEC>,
              (const void *)j3d_pair_kernel<double, CW, RPW, S, true, VEC>},
             {(const void *)j3d_pair_kernel<float, CW, RPW, S, false, VEC>,
              (const void *)j3d_pair_kernel<float, CW, RPW, S, true, VEC>}},
            D::SMEM, {D::W, F::W}, tiles<CW, RPW, S>};
}

}  // namespace

// 100 sweeps on B200 in ms, in this order.  512^3 FP64 26.9 / 30.4 / 27.0 / 31.3, FP32 17.3 / 18.6 / 17.3
// / 18.4; 320^3 FP64 8.1 / 8.4 / 8.1 / 9.2; 256^3 FP64 5.3 / 5.1 / 5.3 / 6.1; 360^3 FP32 7.0 / 6.6 / 7.0 / 6.8;
// 400^3 FP32 12.5 / 11.2 / 12.5 / 13.7.  The first is the default; the second gains where 36 own rows
// fit the grid better than 28; ten stages in place of six change nothing, and three rows per warp
// are never ahead.  All four stay for the autotuner (their indices are part of its interface).
const J3PairShape &j3d_pair_shape(int i, bool vec) {
    static const J3PairShape shapes[J3_PAIR_SHAPES] = {make<8, 4, 6, true>(), make<8, 5, 7, true>(),
                                                       make<8, 4, 10, true>(), make<8, 3, 8, true>()};
    static const J3PairShape ragged = make<8, 5, 7, false>();
    return !vec ? ragged : shapes[i >= 0 && i < J3_PAIR_SHAPES ? i : 0];
}

}  // namespace cfm
