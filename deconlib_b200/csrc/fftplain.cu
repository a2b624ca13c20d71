// The runtime-radix X and column passes (xpass.cuh, colplain.cuh).
#include "colplain.cuh"
#include "xpass.cuh"

namespace dk {

void* pick_xr2c_kernel(int pro) {
    switch (pro) {
        case PRO_ARRAY: return (void*)k_xr2c<PRO_ARRAY>;
        case PRO_CONST: return (void*)k_xr2c<PRO_CONST>;
        case PRO_KERNEL: return (void*)k_xr2c<PRO_KERNEL>;
        case PRO_RLINIT: return (void*)k_xr2c<PRO_RLINIT>;
        case PRO_UP2: return (void*)k_xr2c<PRO_UP2>;
        default: return nullptr;
    }
}

void* pick_xc2r_kernel(int epi) {
    switch (epi) {
        case EPI_STORE: return (void*)k_xc2r<EPI_STORE>;
        case EPI_RL_RATIO: return (void*)k_xc2r<EPI_RL_RATIO>;
        case EPI_RL_UPDATE: return (void*)k_xc2r<EPI_RL_UPDATE>;
        case EPI_PRED: return (void*)k_xc2r<EPI_PRED>;
        case EPI_DOWN2: return (void*)k_xc2r<EPI_DOWN2>;
        default: return nullptr;
    }
}

void* pick_colfft_kernel() { return (void*)k_colfft; }

}  // namespace dk
