// Double-float helpers for FP64-accurate tall-skinny arithmetic on the FP32 pipe
// (GB300 runs FP64 at ~1/64 of the FP32 rate): an FP64 operand is split once
// into an FP32 pair (hi + lo); products are exact to 2^-48 through fma and sums
// carry a compensation term, which keeps ~44 significant bits.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace cg {

// The conversions of the two functions below are calls: in line, the compiler
// predicates them, and they take the FP64 pipe for every value all the same
// (X^T Y of 64 x 8 columns, 2e6 rows: 1.08 ms in line, 0.55 as calls).
static __device__ __noinline__ float2 df_convert(double d) {
  const float h = __double2float_rn(d);
  return make_float2(h, __double2float_rn(d - double(h)));
}
static __device__ __noinline__ double df_convert_up(float f) { return double(f); }

// d = h + l to 2^-49: h the nearest FP32 number, l the nearest to the rest.
// From the bits of d: the conversions and the subtraction run on the FP64 pipe,
// 2 lanes a clock and SM, which bound the kernels that split what they load
// (X C of 64 x 8 columns, 2e6 rows: 0.46 ms, so 0.26; X^T Y 1.39 ms, so 0.55).
// The mantissa's upper 23 bits are rounded by an integer add (ties away from
// zero); the lower 29, sign-extended, are the rest in units of 2^(e - 52).
// Numbers for which h or l would not be a normal FP32 number are converted.
__device__ __forceinline__ void df_split(double d, float& h, float& l) {
  const uint32_t lo = uint32_t(__double2loint(d)), hi = uint32_t(__double2hiint(d));
  const uint32_t mag = hi & 0x7fffffffu, sign = hi & 0x80000000u;
  constexpr uint32_t kLow = (1023u - 70u) << 20, kHigh = (1023u + 127u) << 20;  // 2^-70 <= |d| < 2^127
  const uint32_t rlo = lo + (1u << 28), rhi = mag + (rlo < lo);
  h = __uint_as_float((__funnelshift_l(rlo, rhi, 3) - (896u << 23)) | sign);
  // the lower part as 17 + 12 bits, each made a float by its place in a mantissa
  const int rest = int(lo << 3) >> 3;
  const float top = __uint_as_float(0x4b400000u + uint32_t(rest >> 12)) - 12582912.f;
  const float bot = __uint_as_float(0x4b000000u | uint32_t(rest & 0xfff)) - 8388608.f;
  const float unit = __uint_as_float(((mag & 0x7ff00000u) << 3) - (948u << 23));  // 2^(e - 52)
  l = __uint_as_float(__float_as_uint(fmaf(top, 4096.f, bot) * unit) ^ sign);
  const bool zero = (mag | lo) == 0;  // common (idle lanes, columns not yet filled): no call
  if (zero) {
    h = __uint_as_float(sign);
    l = 0.f;
  }
  if (mag - kLow >= kHigh - kLow && !zero) {
    const float2 p = df_convert(d);
    h = p.x;
    l = p.y;
  }
}

// double(f) from its bits, for sums that leave FP32 (zeros, numbers that are not
// normal and not finite ones apart); X^T Y of FP32 columns 118 -> 110 us
__device__ __forceinline__ double df_widen(float f) {
  const uint32_t u = __float_as_uint(f), sign = u & 0x80000000u, mag = u & 0x7fffffffu;
  double d = __hiloint2double(int(((mag >> 3) + 0x38000000u) | sign), int(u << 29));
  if (mag == 0) d = __hiloint2double(int(sign), 0);
  if (mag - 0x00800000u >= 0x7f000000u && mag) d = df_convert_up(f);
  return d;
}

// (sh, sl) += (ah + al) * (bh + bl), the al * bl term dropped
__device__ __forceinline__ void df_mac(float& sh, float& sl, float ah, float al, float bh, float bl) {
  const float p = ah * bh;
  float e = fmaf(ah, bh, -p);
  e = fmaf(ah, bl, e);
  e = fmaf(al, bh, e);
  const float t = sh + p;
  const float bb = t - sh;
  float err = (sh - (t - bb)) + (p - bb);
  err += sl + e;
  sh = t + err;
  sl = err - (sh - t);
}

// (ah, al) + (bh, bl), compensated
__device__ __forceinline__ void df_add(float& h, float& l, float ah, float al, float bh, float bl) {
  const float s = ah + bh;
  const float bb = s - ah;
  float e = (ah - (s - bb)) + (bh - bb);
  e += al + bl;
  h = s + e;
  l = e - (h - s);
}

}  // namespace cg
