// Instantiations of the register X R2C pass (xreg.cuh), lengths of DK_XREG_LENGTHS_f.
#include "xreg.cuh"

namespace dk {

XRegKernel xreg_r2c_f(int L, int src) {
#define DK_CASE(n) if (L == n) return xreg_r2c_of<n, false>(src);
    DK_XREG_LENGTHS_f(DK_CASE)
#undef DK_CASE
    return XRegKernel{};
}

}  // namespace dk
