// Instantiations of the register X C2R pass (xreg.cuh) on a kx-major spectrum,
// lengths of DK_XREG_LENGTHS_kx.
#include "xreg.cuh"

namespace dk {

XRegKernel xreg_c2r_kx(int L, int epi) {
#define DK_CASE(n) if (L == n) return xreg_c2r_of<n, false, true>(epi);
    DK_XREG_LENGTHS_kx(DK_CASE)
#undef DK_CASE
    return XRegKernel{};
}

}  // namespace dk
