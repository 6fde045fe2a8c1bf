// Codes of the fp8 pages: x * inv rounded to e4m3 (to nearest even, saturating at +-448).
#pragma once
#include <cuda_fp8.h>

#include "common.cuh"

namespace ob {

template <typename T>
__device__ __forceinline__ uint2 to_e4m3x8(const Pack<T>& v, float inv) {
  uint32_t w[2];
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(Elem<T>::to_f(v.v[hh * 4]) * inv, Elem<T>::to_f(v.v[hh * 4 + 1]) * inv),
                                                 __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(Elem<T>::to_f(v.v[hh * 4 + 2]) * inv, Elem<T>::to_f(v.v[hh * 4 + 3]) * inv),
                                                 __NV_SATFINITE, __NV_E4M3);
    w[hh] = lo | (hi << 16);
  }
  return make_uint2(w[0], w[1]);
}

}  // namespace ob
