// The draft map's exponential (draft.cu states the whole contract): y = max(t*log2e, -125); n = rint(y);
// 2^(y-n) by a degree-7 Horner scheme of rounded products and sums; times 2^n.
#pragma once

#include <cuda_runtime.h>

namespace canonical {

__device__ __forceinline__ float exp_canonical(float t) {
  const float y = fmaxf(__fmul_rn(t, __int_as_float(0x3fb8aa3b)), -125.0f);
  const float n = rintf(y);
  const float f = __fsub_rn(y, n);
  float p = __int_as_float(0x377fe5fe);
  p = __fadd_rn(__fmul_rn(p, f), __int_as_float(0x39218489));
  p = __fadd_rn(__fmul_rn(p, f), __int_as_float(0x3aaec3ff));
  p = __fadd_rn(__fmul_rn(p, f), __int_as_float(0x3c1d955b));
  p = __fadd_rn(__fmul_rn(p, f), __int_as_float(0x3d635847));
  p = __fadd_rn(__fmul_rn(p, f), __int_as_float(0x3e75fdf0));
  p = __fadd_rn(__fmul_rn(p, f), __int_as_float(0x3f317218));
  p = __fadd_rn(__fmul_rn(p, f), 1.0f);
  return __fmul_rn(p, __int_as_float((static_cast<int>(n) + 127) << 23));
}

}  // namespace canonical
