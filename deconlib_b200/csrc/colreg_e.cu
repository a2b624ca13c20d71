// Instantiations of the register column pass (colreg.cuh), lengths of DK_PAIR_LENGTHS_E.
#include "colreg.cuh"

namespace dk {

ColRegKernel colreg_group_e(int L, int mode, bool plain) {
#define DK_CASE(n) if (L == n) return colreg_kernel<n>(mode, plain);
    DK_PAIR_LENGTHS_E(DK_CASE)
#undef DK_CASE
    return ColRegKernel{};
}

}  // namespace dk
