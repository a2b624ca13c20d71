// Instantiations of the register PSF passes (psf_passes.cuh), lengths of DK_PAIR_LENGTHS_E.
#include "psf_passes.cuh"

namespace dk {

PsfKernel psf_group_e(int L, bool cols) {
#define DK_CASE(n) if (L == n) return psf_kernel<n>(cols);
    DK_PAIR_LENGTHS_E(DK_CASE)
#undef DK_CASE
    return PsfKernel{};
}

}  // namespace dk
