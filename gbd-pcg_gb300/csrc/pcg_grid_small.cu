// Whole-GPU kernels of one long system for blocks of size n <= 14.
#include "pcg_grid.cuh"
#include "pcg_variants.h"

namespace gbdpcg {
namespace {
template <typename T, int NP, bool PTRI, int G, bool REG>
GridVariant variant() {
    return GridVariant{sizeof(T) == 8, NP, PTRI, G, grid_threads<T, NP, REG>(),
                       (const void *)&pcg_grid_kernel<T, T, NP, PTRI, G, REG>, &SmemPlanGrid<T, T, NP, PTRI>::bytes};
}
// in order of preference: the first that holds a CTA's rows is taken
template <typename T, int NP, bool PTRI>
int kind(GridVariant *out) {
    int c = 0;
    // (a row of three 32 x 32 FP64 blocks leaves a thread no other registers)
    if constexpr (sizeof(T) == 4 || NP <= 24) out[c++] = variant<T, NP, PTRI, 1, true>();
    out[c++] = variant<T, NP, PTRI, 1, false>();
    out[c++] = variant<T, NP, PTRI, 2, false>();
    return c;
}
template <int NP>
int all_of(GridVariant *out) {
    int c = kind<float, NP, false>(out);
    c += kind<float, NP, true>(out + c);
    c += kind<double, NP, false>(out + c);
    c += kind<double, NP, true>(out + c);
    return c;
}
}  // namespace

int variants_grid_small(GridVariant *out) {
    int c = 0;
    c += all_of<6>(out + c);
    c += all_of<8>(out + c);
    c += all_of<12>(out + c);
    c += all_of<14>(out + c);
    return c;
}
}  // namespace gbdpcg
