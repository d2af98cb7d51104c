// Conversions between FP64 and FP32 by integer arithmetic: the values of the
// casts, off the FP64 pipe.  (Only bit casts and integers, so that a host
// compiler can check them against its casts.)
#pragma once

namespace bcfd {

// (float)x by integer arithmetic (round to nearest even): GB300 converts in the
// FP64 pipe, which bounds the residual pass; zeros, and exponents outside
// FP32's normal range by the conversion
__device__ __forceinline__ float to_f32(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned e = (hi >> 20) & 0x7ffu;
  unsigned f = ((hi & 0x7fffffffu) << 3 | lo >> 29) - (896u << 23);
  const unsigned rem = lo & 0x1fffffffu;
  f += (rem > 0x10000000u || (rem == 0x10000000u && (f & 1u))) ? 1u : 0u;
  float r = __uint_as_float((hi & 0x80000000u) | f);
  if (e - 897u >= 254u) r = (float)x;
  return r;
}
// (double)x by integer arithmetic (exact); zeros, subnormals, infinities and
// NaN by the conversion
__device__ __forceinline__ double to_f64(float x) {
  const unsigned u = __float_as_uint(x), e = (u >> 23) & 0xffu;
  double r = __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))), (int)(u << 29));
  if (e - 1u >= 254u) r = (double)x;
  return r;
}

}  // namespace bcfd
