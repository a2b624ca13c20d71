// Instantiations of the register X R2C pass (xreg.cuh) on a kx-major spectrum,
// lengths of DK_XREG_LENGTHS_kx.
#include "xreg.cuh"

namespace dk {

XRegKernel xreg_r2c_kx(int L, int src) {
#define DK_CASE(n) if (L == n) return xreg_r2c_of<n, false, true>(src);
    DK_XREG_LENGTHS_kx(DK_CASE)
#undef DK_CASE
    return XRegKernel{};
}

}  // namespace dk
