// Element-wise passes over arrays, four values per thread and array.
#pragma once

#include <initializer_list>

#include "common.cuh"

namespace dk {

__device__ __forceinline__ int64_t gstride() { return (int64_t)gridDim.x * blockDim.x; }
__device__ __forceinline__ int64_t gtid() { return (int64_t)blockIdx.x * blockDim.x + threadIdx.x; }

// Element-wise loop over n values of NI inputs and NO outputs: groups of four
// with float4 loads and stores when `vec` (every pointer 16-byte aligned),
// then the remainder one by one.  f(in[NI], out[NO]) handles one element;
// a null input reads 0, a null output is not stored; an output may be one of
// the inputs.
template <int NI, int NO, class F>
__device__ __forceinline__ void ew4(int64_t n, const float* const (&in)[NI], float* const (&out)[NO],
                                    bool vec, F&& f) {
    const int64_t ng = vec ? n / 4 : 0;
    for (int64_t gi = gtid(); gi < ng; gi += gstride()) {
        float4 a[NI];
#pragma unroll
        for (int k = 0; k < NI; ++k)
            a[k] = in[k] ? reinterpret_cast<const float4*>(in[k])[gi] : make_float4(0.f, 0.f, 0.f, 0.f);
        float o[NO][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float x[NI], y[NO];
#pragma unroll
            for (int k = 0; k < NI; ++k) x[k] = e == 0 ? a[k].x : e == 1 ? a[k].y : e == 2 ? a[k].z : a[k].w;
            f(x, y);
#pragma unroll
            for (int k = 0; k < NO; ++k) o[k][e] = y[k];
        }
#pragma unroll
        for (int k = 0; k < NO; ++k)
            if (out[k]) reinterpret_cast<float4*>(out[k])[gi] = make_float4(o[k][0], o[k][1], o[k][2], o[k][3]);
    }
    for (int64_t i = 4 * ng + gtid(); i < n; i += gstride()) {
        float x[NI], y[NO];
#pragma unroll
        for (int k = 0; k < NI; ++k) x[k] = in[k] ? in[k][i] : 0.f;
        f(x, y);
#pragma unroll
        for (int k = 0; k < NO; ++k)
            if (out[k]) out[k][i] = y[k];
    }
}

// 1 when every non-null pointer is 16-byte aligned (float4 path of ew4).
inline int al16(std::initializer_list<const void*> ps) {
    for (const void* p : ps)
        if (p && (reinterpret_cast<uintptr_t>(p) & 15) != 0) return 0;
    return 1;
}

}  // namespace dk
