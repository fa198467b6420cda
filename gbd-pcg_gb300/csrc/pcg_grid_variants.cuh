// The whole-GPU kernels of one block-size bound (for pcg_grid_small.cu and
// pcg_grid_large.cu, which share the compile time).
#pragma once
#include "pcg_grid.cuh"
#include "pcg_variants.h"

namespace gbdpcg {

template <typename T, int NP, bool PTRI, int G, bool REG>
GridVariant grid_variant() {
    return GridVariant{sizeof(T) == 8, NP, PTRI, G, grid_threads<T, NP, REG>(),
                       (const void *)&pcg_grid_kernel<T, T, NP, PTRI, G, REG>, &SmemPlanGrid<T, T, NP, PTRI>::bytes};
}
// in order of preference: the first that holds a CTA's rows is taken
template <typename T, int NP, bool PTRI>
int grid_variants_kind(GridVariant *out) {
    int c = 0;
    // (a row of three 32 x 32 FP64 blocks leaves a thread no other registers)
    if constexpr (sizeof(T) == 4 || NP <= 24) out[c++] = grid_variant<T, NP, PTRI, 1, true>();
    out[c++] = grid_variant<T, NP, PTRI, 1, false>();
    out[c++] = grid_variant<T, NP, PTRI, 2, false>();
    return c;
}
template <int NP>
int grid_variants_np(GridVariant *out) {
    int c = grid_variants_kind<float, NP, false>(out);
    c += grid_variants_kind<float, NP, true>(out + c);
    c += grid_variants_kind<double, NP, false>(out + c);
    c += grid_variants_kind<double, NP, true>(out + c);
    return c;
}

}  // namespace gbdpcg
