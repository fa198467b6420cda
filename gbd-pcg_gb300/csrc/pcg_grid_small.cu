// Whole-GPU kernels of one long system for blocks of size n <= 14.
#include "pcg_grid_variants.cuh"

namespace gbdpcg {

int variants_grid_small(GridVariant *out) {
    int c = 0;
    c += grid_variants_np<6>(out + c);
    c += grid_variants_np<8>(out + c);
    c += grid_variants_np<12>(out + c);
    c += grid_variants_np<14>(out + c);
    return c;
}

}  // namespace gbdpcg
