// Whole-GPU kernels of one long system for blocks of size 14 < n <= 32.
#include "pcg_grid_variants.cuh"

namespace gbdpcg {

int variants_grid_large(GridVariant *out) {
    int c = 0;
    c += grid_variants_np<16>(out + c);
    c += grid_variants_np<24>(out + c);
    c += grid_variants_np<32>(out + c);
    return c;
}

}  // namespace gbdpcg
