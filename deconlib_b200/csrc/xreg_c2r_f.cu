// Instantiations of the register X C2R pass (xreg.cuh), lengths of DK_XREG_LENGTHS_f.
#include "xreg.cuh"

namespace dk {

XRegKernel xreg_c2r_f(int L, int epi) {
#define DK_CASE(n) if (L == n) return xreg_c2r_of<n, false>(epi);
    DK_XREG_LENGTHS_f(DK_CASE)
#undef DK_CASE
    return XRegKernel{};
}

}  // namespace dk
