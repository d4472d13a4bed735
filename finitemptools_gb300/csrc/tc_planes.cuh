// Rounding of FP64 / FP32 values to the operand planes of the tensor-core GEMMs: TF32 (hi and, for
// 3xTF32, lo = the rest) or BF16.
#pragma once
#include <cuda_bf16.h>

#include "internal.h"

namespace fmpt {
namespace {

enum { M_TF32 = 0, M_TF32X3 = 1, M_BF16 = 2 };

__device__ __forceinline__ float tf32_rna(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// write one converted value: TF32 (hi, optional lo) or BF16
template <int MODE>
__device__ __forceinline__ void put(void* hi, void* lo, int64_t i, double v) {
  if (MODE == M_BF16) {
    static_cast<__nv_bfloat16*>(hi)[i] = __float2bfloat16_rn(narrow(v));
  } else {
    const float h = tf32_rna(narrow(v));
    static_cast<float*>(hi)[i] = h;
    if (MODE == M_TF32X3) static_cast<float*>(lo)[i] = tf32_rna(narrow(v - widen(h)));
  }
}
// the same of an FP32 value: v - h is exact in FP32 (a multiple of v's last place, below 2^13 of
// them), so no FP64 is needed
template <int MODE>
__device__ __forceinline__ void put(void* hi, void* lo, int64_t i, float v) {
  if (MODE == M_BF16) {
    static_cast<__nv_bfloat16*>(hi)[i] = __float2bfloat16_rn(v);
  } else {
    const float h = tf32_rna(v);
    static_cast<float*>(hi)[i] = h;
    if (MODE == M_TF32X3) static_cast<float*>(lo)[i] = tf32_rna(v - h);
  }
}

}  // namespace
}  // namespace fmpt
