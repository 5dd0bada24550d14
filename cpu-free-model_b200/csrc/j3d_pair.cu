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

const J3PairShape &j3d_pair_shape(int i, bool vec) {
    static const J3PairShape shapes[J3_PAIR_SHAPES] = {make<8, 4, 6, true>(), make<8, 5, 7, true>(),
                                                       make<8, 4, 10, true>(), make<8, 3, 8, true>()};
    static const J3PairShape ragged = make<8, 5, 7, false>();
    return !vec ? ragged : shapes[i >= 0 && i < J3_PAIR_SHAPES ? i : 0];
}

}  // namespace cfm
