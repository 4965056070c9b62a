// Scalar arithmetic of DynamicQuantizeLinear / QuantizeLinear shared by the
// quantize kernels and by the GEMM tail that quantizes its own output.
//
// Semantics follow onnx-mlir's lowering:
//   params    src/Conversion/ONNXToKrnl/Quantization/DynamicQuantizeLinear.cpp:43-84
//   quantize  src/Conversion/ONNXToKrnl/Quantization/QuantizeLinear.cpp:122-145
#pragma once

#include "../common.cuh"

namespace omcuda {

// fp32 arithmetic below uses the _rn intrinsics so that nothing is contracted
// into an fma: the reference emits separate arith ops.
// mode: OMCUDA_MODE_* flags (omcuda.h), the reference's compile-time options
// --disable-quantization-zero-point (zero point 0,
// DynamicQuantizeLinear.cpp:72-83) and enable-fast-math (x * (1 / scale)
// instead of x / scale, QuantizeLinear.cpp:43-44,117-131).
__device__ __forceinline__ void dql_params_from_range(
    float mn, float mx, float *scale, float *zp_f, int mode = 0) {
  float xmax = fmaxf(mx, 0.0f);
  float xmin = fminf(mn, 0.0f);
  float s = __fdiv_rn(__fsub_rn(xmax, xmin), 255.0f);
  float inter = __fsub_rn(0.0f, __fdiv_rn(xmin, s));
  float z = round_even(clipf(inter, 0.0f, 255.0f));
  *scale = s;
  *zp_f = (mode & OMCUDA_MODE_NO_ZERO_POINT) ? 0.0f : z;
}

// One element exactly as the reference computes it
// (QuantizeLinear.cpp:124-145): IEEE divide, round half even, add the zero
// point, clip, convert.
template <bool kSigned>
__device__ __forceinline__ uint32_t quantize_quotient(float q, float zp_f);
template <bool kSigned>
__device__ __forceinline__ uint32_t quantize_one_exact(
    float x, float scale, float zp_f, bool use_rcp = false) {
  return quantize_quotient<kSigned>(
      use_rcp ? __fmul_rn(x, __fdiv_rn(1.0f, scale)) : __fdiv_rn(x, scale), zp_f);
}
template <bool kSigned>
__device__ __forceinline__ uint32_t quantize_quotient(float q, float zp_f) {
  float r = round_even(q);
  float a = __fadd_rn(r, zp_f);
  if (kSigned) {
    float s = clipf(a, -128.0f, 127.0f);
    return (uint32_t)(int32_t)s & 0xffu; // fptosi, then trunc to 8 bits
  }
  float s = clipf(a, 0.0f, 255.0f);
  return (uint32_t)s; // fptoui; already within 8 bits
}

// Per-launch constants of the fast path.
struct QuantConsts {
  float scale, rcp, zp_f;
  float fix; // what a residual of the quotient is multiplied by: rcp, or 0
  float x_lo, x_hi; // inputs beyond these saturate
  bool fast;
  bool use_rcp; // fast-math mode: the reference multiplies by RN(1 / scale)
};

// The smallest and the largest result; integers up to 2^22 on either side of
// kQuantMagic lie in the low mantissa bits of a float that has it added.
template <bool kSigned>
struct QuantBounds {
  static constexpr float lo = kSigned ? -128.0f : 0.0f;
  static constexpr float hi = kSigned ? 127.0f : 255.0f;
};
constexpr float kQuantMagic = 12582912.0f; // 1.5 * 2^23

template <bool kSigned>
__device__ __forceinline__ QuantConsts make_quant_consts(
    float scale, float zp_f, int mode = 0) {
  QuantConsts c;
  c.scale = scale;
  c.zp_f = (mode & OMCUDA_MODE_NO_ZERO_POINT) ? 0.0f : zp_f;
  c.use_rcp = (mode & OMCUDA_MODE_FAST_MATH) != 0;
  c.rcp = __fdiv_rn(1.0f, scale);
  c.fix = c.use_rcp ? 0.0f : c.rcp;
  // A quarter beyond the last integer: a clamped input still rounds to it.
  c.x_lo = __fmul_rn(QuantBounds<kSigned>::lo - c.zp_f - 0.25f, scale);
  c.x_hi = __fmul_rn(QuantBounds<kSigned>::hi - c.zp_f + 0.25f, scale);
  // The shortcut needs a normal, finite reciprocal and residuals that do not
  // underflow; anything else (scale 0 from an all-zero tensor, negative,
  // denormal or huge scales) takes another path to the same results.
  c.fast = (scale > 1e-30f) && (scale < 1e30f);
  return c;
}

// The quotients x / scale of two values, rounded as the IEEE divide rounds them,
// by multiplications only (Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", 1990): with y = RN(1/scale), one
// correction q + (x - q scale) y of q = RN(x y) leaves it within an ulp of the
// quotient, and from such a q the same correction gives RN(x / scale).  The
// second residual is exact, as that asks: with |q| >= 1/4 (anything smaller
// rounds to zero whatever its last bits are) and scale > 1e-30 its last bit is
// at least 2^-149.
// In fast-math mode the reference's quotient is RN(x y) itself: the corrections then
// multiply the residuals, which are finite, by zero.
__device__ __forceinline__ uint64_t quotient_x2(uint64_t x, const QuantConsts &c) {
  const uint64_t y = pack_f32x2(c.rcp, c.rcp), ns = pack_f32x2(-c.scale, -c.scale);
  const uint64_t fix = pack_f32x2(c.fix, c.fix);
  uint64_t q = mul_f32x2(x, y);
  q = fma_f32x2(fma_f32x2(q, ns, x), fix, q);
  return fma_f32x2(fma_f32x2(q, ns, x), fix, q);
}

// Inputs that saturate, cut back to where they still do (a NaN goes to the lower
// bound, where maxnum/minnum send it in the reference as well).
__device__ __forceinline__ float quant_clamp(float x, const QuantConsts &c) {
  return fminf(fmaxf(x, c.x_lo), c.x_hi);
}

// Four elements by the exact formula, out of line: scales the fast path below
// does not take.
template <bool kSigned>
__device__ __noinline__ uint32_t quantize_four_exact(
    float4 v, float scale, float zp_f, bool use_rcp) {
  return quantize_one_exact<kSigned>(v.x, scale, zp_f, use_rcp) |
         (quantize_one_exact<kSigned>(v.y, scale, zp_f, use_rcp) << 8) |
         (quantize_one_exact<kSigned>(v.z, scale, zp_f, use_rcp) << 16) |
         (quantize_one_exact<kSigned>(v.w, scale, zp_f, use_rcp) << 24);
}

// Same result as quantize_one_exact on the four elements of a float4, with no
// divide or convert instruction and no branch per element: the quotient as
// above, rounded half-even by adding kQuantMagic, the zero point added to that,
// and the result is the low byte (two's complement for the signed type) of the
// mantissa.  About six arithmetic instructions an element; with the moves in and out of
// packed pairs, predicates, addresses and the fold of the partials quantize_kernel executed 18 on
// 16 Mi values, which are quantize_wide_kernel's now: 8.5.  (An approximate quotient with
// the exact divide for elements near a tie costs less on paper, but with a test
// at 0.499 a fifth of the warps had such an element among their 128 and took the
// divide: 16 Mi values 16.4 us, 7.3 without any arithmetic.)
template <bool kSigned>
__device__ __forceinline__ uint32_t quantize_four_fast(float4 v, const QuantConsts &c) { // c.fast
  const uint64_t magic = pack_f32x2(kQuantMagic, kQuantMagic);
  const uint64_t zp = pack_f32x2(c.zp_f, c.zp_f);
  const uint64_t q01 = quotient_x2(pack_f32x2(quant_clamp(v.x, c), quant_clamp(v.y, c)), c);
  const uint64_t q23 = quotient_x2(pack_f32x2(quant_clamp(v.z, c), quant_clamp(v.w, c)), c);
  const uint64_t t01 = add_f32x2(add_f32x2(q01, magic), zp);
  const uint64_t t23 = add_f32x2(add_f32x2(q23, magic), zp);
  const uint32_t b01 = __byte_perm((uint32_t)t01, (uint32_t)(t01 >> 32), 0x0040);
  const uint32_t b23 = __byte_perm((uint32_t)t23, (uint32_t)(t23 >> 32), 0x0040);
  return __byte_perm(b01, b23, 0x5410);
}
template <bool kSigned>
__device__ __forceinline__ uint32_t quantize_four(float4 v, const QuantConsts &c) {
  if (!c.fast)
    return quantize_four_exact<kSigned>(v, c.scale, c.zp_f, c.use_rcp);
  return quantize_four_fast<kSigned>(v, c);
}

template <bool kSigned>
__device__ __forceinline__ uint32_t quantize_one(float x, const QuantConsts &c) {
  if (!c.fast)
    return quantize_one_exact<kSigned>(x, c.scale, c.zp_f, c.use_rcp);
  return quantize_four<kSigned>(make_float4(x, x, x, x), c) & 0xffu;
}

} // namespace omcuda
