// DynamicQuantizeLinear / QuantizeLinear / DequantizeLinear kernels.
//
// Semantics follow onnx-mlir's lowering:
//   min/max   src/Conversion/ONNXToKrnl/Math/Reduction.cpp:394-548 (minnum/maxnum,
//             identities +inf/-inf)
//   params    src/Conversion/ONNXToKrnl/Quantization/DynamicQuantizeLinear.cpp:43-84
//   quantize  src/Conversion/ONNXToKrnl/Quantization/QuantizeLinear.cpp:122-145
//   dequant   src/Conversion/ONNXToKrnl/Math/Elementwise.cpp:1438-1461
//
// Layout: tensors are flat, dense, row-major.  What one cluster holds in its
// registers is one launch (dql_small_kernel).  Above that the reduction leaves
// one partial {min, max} per block in scratch, and every block of the quantize
// pass, a second launch, folds them all while its first values are on their way:
// nobody draws a ticket or waits for another block, and the scratch needs no
// initial value.
#include <cooperative_groups.h>

#include "../common.cuh"
#include "../runtime/internal.h"
#include "quantize.cuh"

namespace cg = cooperative_groups;

namespace omcuda {

static constexpr int kDqlThreads = 256;
static constexpr int kQuantUnroll = 4;
static constexpr int kSingleUnroll = 4; // values in flight where a thread takes single ones
// The reduction's blocks, and so the partials every block of the pass behind it
// folds: four of 512 threads fill an SM.
static constexpr int kRangeThreads = 512;
static constexpr int kRangeFewThreads = 128; // of the blocks for few values
static constexpr int kRangeBlocksPerSm = 4;
static constexpr int kRangeUnroll = 8;
static constexpr int kRangeMaxParts = 2048;

// What a caller's scratch holds: 64 bytes that are left alone (callers may keep
// them zero, as they once had to be) and the partials, at the next address
// that takes 8-byte accesses.
static constexpr int64_t kScratchBytes = 64 + 8 + (int64_t)kRangeMaxParts * sizeof(float2);
static float2 *scratch_parts(void *scratch) {
  return reinterpret_cast<float2 *>(((uintptr_t)scratch + 64 + 7) & ~(uintptr_t)7);
}

// The extremes over a block of kThreads threads, in every thread.
template <int kThreads>
__device__ __forceinline__ void block_range(float &lo, float &hi) {
  __shared__ float s_lo[kThreads / 32], s_hi[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  lo = warp_min(lo);
  hi = warp_max(hi);
  if (lane == 0) {
    s_lo[warp] = lo;
    s_hi[warp] = hi;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) {
    lo = fminf(lo, s_lo[w]);
    hi = fmaxf(hi, s_hi[w]);
  }
}

// Bound by the read of x: 64 Mi values in 39 us (6.9 TB/s), 16 Mi that lie in L2 in
// 6 (11 TB/s).  Plain loads and not streaming ones: the quantize pass finds in
// L2 what still fits there.  kFull: the run is kRangeUnroll float4 a thread, known to
// the compiler (64 Mi values 104 us the whole call without that, 101 with).  kZero: sets the
// `zeros` words of `sums` to zero as well, for a pass behind it that adds to them.  kDeep:
// registers for all loads of a run at once.  With the 32 of a full SM the compiler makes two or
// three round trips of them, all that a few blocks have to do: linear 128 x 4096 x 4096 17.9 ->
// 15.3 us, 64 x 8192 x 8192 24.3 -> 22.0, 700 x 768 x 768 11.3 -> 10.3, 777 x 1001 x 1537 17.3 -> 16.2;
// DynamicQuantizeLinear of 600000 values 5.2 -> 4.6, 6 M 11.9 -> 10.8, 64 Mi 92.9 -> 90.8 (all on the
// same values call after call, of which L2 keeps some).
template <bool kFull, bool kZero, int kThreads, bool kDeep>
__global__ void __launch_bounds__(kThreads, kDeep ? 1024 / kThreads : 2048 / kThreads)
    dql_minmax_kernel(const float *__restrict__ x, int64_t n, float2 *__restrict__ part,
        int unroll, int32_t *__restrict__ sums, int zeros) {
  pdl_sync();
  x = after_pdl(x);
  if (kZero)
    for (int i = blockIdx.x * kThreads + threadIdx.x; i < zeros;
         i += gridDim.x * kThreads)
      sums[i] = 0;
  float lo = INFINITY, hi = -INFINITY;
  const bool aligned = ((uintptr_t)x & 15u) == 0;
  const int64_t n4 = aligned ? n >> 2 : 0;
  const float4 *x4 = reinterpret_cast<const float4 *>(x);
  // what is left of a group of four, or everything when x is not aligned; the
  // first of it is asked for now and not behind the rest
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  int64_t j = (n4 << 2) + tid;
  float tail = j < n ? __ldg(x + j) : 0.0f;
  const int run = (kFull ? kRangeUnroll : unroll) * kThreads;
  for (int64_t base = (int64_t)blockIdx.x * run + threadIdx.x; base < n4;
       base += (int64_t)gridDim.x * run) {
    // (what lies past the end counts as zero, which changes neither scalar: the
    // range is widened to hold 0 before anything is derived from it)
    float4 v[kRangeUnroll];
#pragma unroll
    for (int u = 0; u < kRangeUnroll; ++u)
      v[u] = (kFull || u < unroll) && base + u * kThreads < n4
                 ? __ldg(x4 + base + u * kThreads)
                 : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int u = 0; u < kRangeUnroll; ++u) {
      lo = min3f(min3f(lo, v[u].x, v[u].y), v[u].z, v[u].w);
      hi = max3f(max3f(hi, v[u].x, v[u].y), v[u].z, v[u].w);
    }
  }
  lo = fminf(lo, tail);
  hi = fmaxf(hi, tail);
#pragma unroll 8
  for (j += nthreads; j < n; j += nthreads) {
    const float f = __ldg(x + j);
    lo = fminf(lo, f);
    hi = fmaxf(hi, f);
  }
  block_range<kThreads>(lo, hi);
  if (threadIdx.x == 0)
    part[blockIdx.x] = make_float2(lo, hi);
}

// The extremes that the reduction's blocks left, in every thread of the block.
struct RangeParts {
  const float2 *part;
  int count;
};
__device__ __forceinline__ void fold_parts(const RangeParts &r, float &lo, float &hi) {
  const float2 *part = after_pdl(r.part);
  lo = INFINITY;
  hi = -INFINITY;
  for (int i = threadIdx.x; i < r.count; i += kDqlThreads) {
    const float2 q = __ldg(part + i);
    lo = fminf(lo, q.x);
    hi = fmaxf(hi, q.y);
  }
  block_range<kDqlThreads>(lo, hi);
}

// Folds the min / max of x into a running range (the encoding and the commit
// rule of range_commit_warp): the reduction of DynamicQuantizeLinear in the
// form the producers of the encoder harness use, for a tensor that has no
// producer on the device.
__global__ void __launch_bounds__(kDqlThreads)
    range_fold_kernel(const float *__restrict__ x, int64_t n, uint32_t *__restrict__ range) {
  float lo = INFINITY, hi = -INFINITY;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  if ((((uintptr_t)x) & 15u) == 0) {
    const int64_t n4 = n >> 2;
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    for (int64_t i = tid; i < n4; i += nthreads) {
      const float4 a = __ldcs(x4 + i);
      lo = fminf(lo, fminf(fminf(a.x, a.y), fminf(a.z, a.w)));
      hi = fmaxf(hi, fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)));
    }
    for (int64_t j = (n4 << 2) + tid; j < n; j += nthreads) {
      lo = fminf(lo, x[j]);
      hi = fmaxf(hi, x[j]);
    }
  } else {
    for (int64_t j = tid; j < n; j += nthreads) {
      lo = fminf(lo, x[j]);
      hi = fmaxf(hi, x[j]);
    }
  }
  range_commit_warp(range, lo, hi);
}

// Where the range-driven forms of the kernel leave their scalars; each may be null.
struct QuantOutputs {
  float *params;  // {scale, zero point as float}
  float *y_scale; // the op's y_scale output
  uint8_t *y_zp;  // the op's y_zero_point output

  __device__ void publish(float scale, float zp_f) const {
    if (params) {
      params[0] = scale;
      params[1] = zp_f;
    }
    if (y_scale)
      *y_scale = scale;
    if (y_zp)
      *y_zp = (uint8_t)(unsigned int)zp_f; // fptoui; zp_f is in [0,255]
  }
};

// What a quantize pass takes its scale and zero point from: as DynamicQuantizeLinear
// derives them from `parts` (count > 0: the reduction's partials) or from `range` (a
// producer's running {min,max}, ordered-uint encoding, see f32_to_ordered), or
// the given scale and 8-bit zero point (zp8 may be null).
struct QuantSource {
  RangeParts parts;
  const uint32_t *range;
  const float *scale;
  const void *zp8;
};
// zeros: set where the reduction has seen nothing but zeros (and NaNs) in x.
template <bool kSigned>
__device__ __forceinline__ QuantConsts quant_scalars(
    const QuantSource &src, const QuantOutputs &outs, int mode, bool *zeros = nullptr) {
  float scale, zp_f;
  if (src.parts.count > 0 || src.range) {
    // (every thread derives the same two scalars)
    float lo, hi;
    if (src.parts.count > 0) {
      fold_parts(src.parts, lo, hi);
      if (zeros)
        *zeros = lo >= 0.0f && hi <= 0.0f;
    } else {
      const uint32_t *range = after_pdl(src.range);
      lo = ordered_to_f32(__ldg(range));
      hi = ordered_to_f32(__ldg(range + 1));
    }
    dql_params_from_range(lo, hi, &scale, &zp_f, mode);
    if (blockIdx.x == 0 && threadIdx.x == 0)
      outs.publish(scale, zp_f);
  } else {
    scale = __ldg(after_pdl(src.scale));
    const void *zp8 = after_pdl(src.zp8);
    if (!zp8)
      zp_f = 0.0f;
    else if (kSigned)
      zp_f = (float)*reinterpret_cast<const int8_t *>(zp8);
    else
      zp_f = (float)*reinterpret_cast<const uint8_t *>(zp8);
  }
  return make_quant_consts<kSigned>(scale, zp_f, mode);
}

// x 16-byte and y 4-byte aligned.
template <bool kSigned>
__global__ void __launch_bounds__(kDqlThreads)
    quantize_kernel(const float *__restrict__ x, int64_t n, uint8_t *__restrict__ y,
        QuantSource src, QuantOutputs outs, int mode, int unroll) {
  pdl_sync();
  x = after_pdl(x);
  // A block takes runs of unroll * 256 neighbouring float4 (16 KiB at most), the
  // loads of the first before it derives the scalars: three dependent divides
  // that a launch on a small tensor would otherwise spend before it asks for data.
  // Runs and not a stride of the whole grid, and only four loads in flight per
  // thread so that more blocks fit: 64 Mi values 67.0 -> 64.1 us, an encoder run of
  // 1 x 61 resident tokens 741 -> 659 us, of 32 x 128 1903 -> 1839.
  const int64_t n4 = n >> 2;
  const float4 *x4 = reinterpret_cast<const float4 *>(x);
  uint32_t *y4 = reinterpret_cast<uint32_t *>(y);
  const int run = unroll * kDqlThreads;
  int64_t base = (int64_t)blockIdx.x * run + threadIdx.x;
  float4 v[kQuantUnroll];
#pragma unroll
  for (int u = 0; u < kQuantUnroll; ++u)
    if (u < unroll && base + u * kDqlThreads < n4)
      v[u] = __ldcs(x4 + base + u * kDqlThreads);
  // what is left of a word
  const int64_t rest = (n4 << 2) + threadIdx.x;
  const bool takes_rest = blockIdx.x == 0 && rest < n;
  const float last = takes_rest ? __ldg(x + rest) : 0.0f;
  const QuantConsts qc = quant_scalars<kSigned>(src, outs, mode);
  while (base < n4) {
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u)
      if (u < unroll && base + u * kDqlThreads < n4)
        y4[base + u * kDqlThreads] = quantize_four<kSigned>(v[u], qc);
    base += (int64_t)gridDim.x * run;
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u)
      if (u < unroll && base + u * kDqlThreads < n4)
        v[u] = __ldcs(x4 + base + u * kDqlThreads);
  }
  if (takes_rest)
    y[rest] = (uint8_t)quantize_one<kSigned>(last, qc);
}

// Eight neighbouring values, p 32-byte aligned.  kOnce: they are not asked for again soon, L2
// may let go of them first.
struct Eight {
  float4 a, b;
};
template <bool kOnce>
__device__ __forceinline__ Eight load_eight(const float *p) {
  Eight v;
  if (kOnce)
    asm volatile("ld.global.L1::no_allocate.L2::evict_first.v8.f32 {%0, %1, %2, %3, %4, %5, %6, "
                 "%7}, [%8];"
                 : "=f"(v.a.x), "=f"(v.a.y), "=f"(v.a.z), "=f"(v.a.w), "=f"(v.b.x), "=f"(v.b.y),
                   "=f"(v.b.z), "=f"(v.b.w)
                 : "l"(p));
  else
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v.a.x), "=f"(v.a.y), "=f"(v.a.z), "=f"(v.a.w), "=f"(v.b.x), "=f"(v.b.y),
                   "=f"(v.b.z), "=f"(v.b.w)
                 : "l"(p));
  return v;
}

// The pass by the exact formula, for scales quantize_four_fast does not take.  Out of line, as
// the kernel below is short of registers.  A scale of zero leaves three quotients, by the sign of
// x.  It does not say that x is zero: the 255th part of a range of up to 127 steps of the least
// denormal is zero too, and such values are divided to infinities, not to the NaN of 0 / 0.
// zeros, as quant_scalars has it, does say so, and x is not read.  (DynamicQuantizeLinear, value by
// value and so: 300000 zeros 5.7 and 4.7 us, 64 Mi 188 and 66; 64 Mi denormals 212 and 98.)
template <bool kSigned>
__device__ __noinline__ void quantize_pass_exact(
    const float *x, int64_t n, uint8_t *y, float scale, float zp_f, bool use_rcp, bool zeros) {
  const int64_t step = (int64_t)gridDim.x * kDqlThreads, n4 = n >> 2;
  const int64_t tid = (int64_t)blockIdx.x * kDqlThreads + threadIdx.x;
  const float4 *x4 = reinterpret_cast<const float4 *>(x);
  uint32_t *y4 = reinterpret_cast<uint32_t *>(y);
  const int64_t j = (n4 << 2) + tid; // what is left of a group of four
  if (scale == 0.0f) {
    const float inf = __fdiv_rn(1.0f, scale); // (of the sign of scale)
    const uint32_t q0 = quantize_quotient<kSigned>(__fmul_rn(0.0f, inf), zp_f); // a NaN's too
    const uint32_t qp = quantize_quotient<kSigned>(inf, zp_f);
    const uint32_t qn = quantize_quotient<kSigned>(-inf, zp_f);
    if (zeros) {
#pragma unroll 1
      for (int64_t i = tid; i < n4; i += step)
        y4[i] = q0 * 0x01010101u;
      if (j < n)
        y[j] = (uint8_t)q0;
      return;
    }
    const auto one = [&](float f) { return f > 0.0f ? qp : f < 0.0f ? qn : q0; };
#pragma unroll 4
    for (int64_t i = tid; i < n4; i += step) {
      const float4 v = __ldg(x4 + i);
      y4[i] = one(v.x) | one(v.y) << 8 | one(v.z) << 16 | one(v.w) << 24;
    }
    if (j < n)
      y[j] = (uint8_t)one(__ldg(x + j));
    return;
  }
  const float rcp = __fdiv_rn(1.0f, scale);
  if (fabsf(scale) < INFINITY && (!use_rcp || fabsf(rcp) < INFINITY)) {
    // The sign and a power of two that go into x as well leave the quotients as they are (what of x
    // it takes below 2^-126 has a quotient below 2^-62) and make the scale one of quantize_four_fast's.
    // Fast-math mode's reciprocal is that of the scale as it is, rounded where it is a denormal.
    // (Values of 1e-30, DynamicQuantizeLinear: 300000 in the 16-byte pass 5.6 us, here divided one
    // by one 8.6, so 5.0; 64 Mi 229, 248 and 103; 24000 from a range 2.8, 6.1 and 2.6.  A given scale
    // of -0.05, the same three: 300000 2.5, 4.4 and 2.5, 64 Mi 91, 146 and 80; in fast-math mode 2.2, 3.7
    // and 2.5, 84, 135 and 80.)
    const float f = copysignf(fabsf(scale) < 1.0f ? 0x1p64f : 0x1p-64f, scale);
    QuantConsts qc = make_quant_consts<kSigned>(
        __fmul_rn(scale, f), zp_f, use_rcp ? OMCUDA_MODE_FAST_MATH : 0);
    if (use_rcp)
      qc.rcp = __fmul_rn(rcp, copysignf(fabsf(scale) < 1.0f ? 0x1p-64f : 0x1p64f, scale));
#pragma unroll 2
    for (int64_t i = tid; i < n4; i += step) {
      const float4 v = __ldg(x4 + i);
      y4[i] = quantize_four_fast<kSigned>(
          make_float4(__fmul_rn(v.x, f), __fmul_rn(v.y, f), __fmul_rn(v.z, f), __fmul_rn(v.w, f)), qc);
    }
    if (j < n) {
      const float e = __fmul_rn(__ldg(x + j), f);
      y[j] = (uint8_t)quantize_four_fast<kSigned>(make_float4(e, e, e, e), qc);
    }
    return;
  }
  // What is left are products by 0 (an infinite scale, also by definition), an infinity or a NaN.
  // (An infinite scale: 64 Mi in the 16-byte pass 143 us, divided one by one 202, so 83.)
  const auto one = [&](float f) { return quantize_quotient<kSigned>(__fmul_rn(f, rcp), zp_f); };
#pragma unroll 4
  for (int64_t i = tid; i < n4; i += step) {
    const float4 v = __ldg(x4 + i);
    y4[i] = one(v.x) | one(v.y) << 8 | one(v.z) << 16 | one(v.w) << 24;
  }
  if (j < n)
    y[j] = (uint8_t)one(__ldg(x + j));
}

// quantize_kernel's pass for many values, x 32-byte and y 8-byte aligned.  That kernel takes what
// lies in L2 hardly faster than what comes from HBM (16 Mi values 11.5 us, 7.4 without its
// arithmetic): it executes 72 instructions per float4, half of them predicates and 64-bit
// addresses.  Here runs are whole (what is left goes group by group), the addresses of a
// run are one pointer and constants, a load is 32 bytes a lane and a store 8.  Two groups a
// thread: four take 79 registers, three blocks per SM and no less time.  Whole calls
// on values that change from call to call, before this pass and the deeper loads of the reduction
// and now: DynamicQuantizeLinear of 1 Mi values 6.0 -> 5.7 us, 6 M 13.1 -> 10.7, 16 Mi 28.8 -> 23.6,
// 64 Mi 102.5 -> 93.7 (9 bytes a value: 6.4 TB/s), 128 Mi 208 -> 183; a given scale 2 M 3.5 -> 3.0,
// 64 Mi 58.1 -> 53.3.
constexpr int kWideGroups = 2;
// Resident at once.  (Five leave 51 registers, and what then goes to memory costs
// DynamicQuantizeLinear of 64 Mi 102 us instead of 92, the same values call after call.)
constexpr int kWideBlocksPerSm = 4;
template <bool kSigned, bool kOnce>
__global__ void __launch_bounds__(kDqlThreads, kWideBlocksPerSm)
    quantize_wide_kernel(const float *__restrict__ x, int64_t n, uint8_t *__restrict__ y,
        QuantSource src, QuantOutputs outs, int mode) {
  pdl_sync();
  x = after_pdl(x);
  constexpr int kGroups = kWideGroups, kRun = kGroups * kDqlThreads;
  const int64_t n8 = n >> 3;
  const unsigned runs = (unsigned)(n8 / kRun);
  unsigned r = blockIdx.x;
  const float *xr = x + ((int64_t)r * kRun + threadIdx.x) * 8;
  Eight v[kGroups];
  if (r < runs)
#pragma unroll
    for (int u = 0; u < kGroups; ++u)
      v[u] = load_eight<kOnce>(xr + u * (kDqlThreads * 8));
  bool zeros = false;
  const QuantConsts qc = quant_scalars<kSigned>(src, outs, mode, &zeros);
  if (!qc.fast) {
    quantize_pass_exact<kSigned>(x, n, y, qc.scale, qc.zp_f, qc.use_rcp, zeros);
    return;
  }
  uint2 *yr = reinterpret_cast<uint2 *>(y) + ((int64_t)r * kRun + threadIdx.x);
  while (r < runs) {
    uint2 w[kGroups];
#pragma unroll
    for (int u = 0; u < kGroups; ++u)
      w[u] = make_uint2(
          quantize_four_fast<kSigned>(v[u].a, qc), quantize_four_fast<kSigned>(v[u].b, qc));
    uint2 *const out = yr;
    r += gridDim.x;
    xr += (int64_t)gridDim.x * (kRun * 8);
    yr += (int64_t)gridDim.x * kRun;
    if (r < runs)
#pragma unroll
      for (int u = 0; u < kGroups; ++u)
        v[u] = load_eight<kOnce>(xr + u * (kDqlThreads * 8));
#pragma unroll
    for (int u = 0; u < kGroups; ++u)
      out[u * kDqlThreads] = w[u];
  }
  // what is left, from the last block on: those have the fewest runs
  const unsigned b = gridDim.x - 1 - blockIdx.x;
#pragma unroll 1
  for (int64_t g = (int64_t)runs * kRun + (int64_t)b * kDqlThreads + threadIdx.x; g < n8;
       g += (int64_t)gridDim.x * kDqlThreads) {
    const Eight e = load_eight<kOnce>(x + 8 * g);
    reinterpret_cast<uint2 *>(y)[g] =
        make_uint2(quantize_four_fast<kSigned>(e.a, qc), quantize_four_fast<kSigned>(e.b, qc));
  }
  const int64_t j = (n8 << 3) + threadIdx.x;
  if (b == 0 && j < n) {
    const float f = __ldg(x + j);
    y[j] = (uint8_t)quantize_four_fast<kSigned>(make_float4(f, f, f, f), qc);
  }
}

// The same one value at a time, for tensors that are not aligned so.  A kernel of
// its own, as for dequantize: the loads of several trips together take registers
// that the one above would miss (in it, 64 Mi aligned values went from 54 to 57 us),
// and one value asked for ahead of the one in work is too little to hide memory
// behind.  64 Mi values quantized 224 -> 109 us, dynamically 365 -> 159, 1 Mi 6.1 ->
// 3.5 and 13.1 -> 8.8, on resident blocks and with four loads together.
template <bool kSigned>
__global__ void __launch_bounds__(kDqlThreads)
    quantize_single_kernel(const float *__restrict__ x, int64_t n, uint8_t *__restrict__ y,
        QuantSource src, QuantOutputs outs, int mode) {
  pdl_sync();
  x = after_pdl(x);
  const int64_t step = (int64_t)gridDim.x * kDqlThreads;
  int64_t j = (int64_t)blockIdx.x * kDqlThreads + threadIdx.x;
  const float first = j < n ? __ldg(x + j) : 0.0f;
  const QuantConsts qc = quant_scalars<kSigned>(src, outs, mode);
  if (j >= n)
    return;
  y[j] = (uint8_t)quantize_one<kSigned>(first, qc);
  for (j += step; j < n; j += kSingleUnroll * step) {
    float f[kSingleUnroll];
#pragma unroll
    for (int u = 0; u < kSingleUnroll; ++u)
      if (j + u * step < n)
        f[u] = __ldg(x + j + u * step);
#pragma unroll
    for (int u = 0; u < kSingleUnroll; ++u)
      if (j + u * step < n)
        y[j + u * step] = (uint8_t)quantize_one<kSigned>(f[u], qc);
  }
}

// The quantize pass by rows, written in the aligned rows the GEMM kernels take
// (zero from cols up to pitch), with the sums of the quantized rows where the
// weight has a zero point.  kWarps warps make a row at a time: one while that
// keeps the machine busy, for there is nothing to wait for then, else a block, and
// where the rows are few, `split` blocks, whose sums are added up in memory that the
// reduction has cleared.  A thread makes one output word from four neighbouring
// values, four words in flight.  The linear 777 x 1001 x 1537 22.5 -> 17.5 us
// together with the reduction above, 777 x 1024 x 1536 19.8 -> 14.3.
constexpr int kRowsUnroll = 4;
template <int kWarps, bool kSplit>
__global__ void __launch_bounds__(kDqlThreads)
    quantize_rows_kernel(const float *__restrict__ x, int64_t rows, int cols, int pitch,
        uint8_t *__restrict__ y, int32_t *__restrict__ rowsum, RangeParts parts,
        QuantOutputs outs, int vec_in, int split, int mode) {
  pdl_sync();
  x = after_pdl(x);
  constexpr int kThreads = 32 * kWarps, kRows = kDqlThreads / kThreads;
  __shared__ int32_t part[kDqlThreads / 32];
  float lo, hi, scale, zp_f;
  fold_parts(parts, lo, hi);
  dql_params_from_range(lo, hi, &scale, &zp_f, mode);
  if (blockIdx.x == 0 && threadIdx.x == 0)
    outs.publish(scale, zp_f);
  const QuantConsts qc = make_quant_consts<false>(scale, zp_f, mode);
  const int t = threadIdx.x % kThreads, warp = threadIdx.x >> 5;
  const int words = pitch >> 2;
  // (a split row: every grid has a block for each part of it)
  const int step = kSplit ? split * kThreads : kThreads; // words apart
  const int first = kSplit ? (int)(blockIdx.x % (unsigned)split) * kThreads + t : t;
  for (int64_t r = kSplit ? (int64_t)(blockIdx.x / (unsigned)split)
                          : (int64_t)blockIdx.x * kRows + threadIdx.x / kThreads;
       r < rows; r += kSplit ? rows : (int64_t)gridDim.x * kRows) {
    const float *xr = x + r * cols;
    uint32_t *yr = reinterpret_cast<uint32_t *>(y + r * pitch);
    int32_t sum = 0;
    for (int j0 = first; j0 < words; j0 += kRowsUnroll * step) {
      float4 v[kRowsUnroll];
#pragma unroll
      for (int u = 0; u < kRowsUnroll; ++u) {
        const int c = 4 * (j0 + u * step), have = cols - c;
        v[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (have >= 4 && vec_in) {
          v[u] = __ldcs(reinterpret_cast<const float4 *>(xr + c));
        } else {
          if (have > 0)
            v[u].x = __ldg(xr + c);
          if (have > 1)
            v[u].y = __ldg(xr + c + 1);
          if (have > 2)
            v[u].z = __ldg(xr + c + 2);
          if (have > 3)
            v[u].w = __ldg(xr + c + 3);
        }
      }
#pragma unroll
      for (int u = 0; u < kRowsUnroll; ++u) {
        const int j = j0 + u * step, have = cols - 4 * j;
        if (j >= words)
          break;
        uint32_t w = have > 0 ? quantize_four<false>(v[u], qc) : 0u;
        if (have > 0 && have < 4)
          w &= (1u << (8 * have)) - 1u;
        yr[j] = w;
        sum = add_bytes<false>(w, sum);
      }
    }
    if (!rowsum)
      continue;
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (kWarps == 1) {
      if (t == 0)
        rowsum[r] = sum;
    } else {
      __syncthreads(); // part[] of the row before has been read
      if ((threadIdx.x & 31) == 0)
        part[warp] = sum;
      __syncthreads();
      if (threadIdx.x == 0) {
        int32_t s = 0;
        for (int w = 0; w < kDqlThreads / 32; ++w)
          s += part[w];
        if (kSplit)
          atomicAdd(rowsum + r, s);
        else
          rowsum[r] = s;
      }
    }
  }
}

// DynamicQuantizeLinear of a tensor of which every thread of one cluster holds
// kWords words of four values: what bounds small tensors is launches and round trips
// through memory.  Here every thread loads its values once, the CTAs exchange their
// {min,max} through distributed shared memory, every thread derives the two
// scalars and quantizes what it still holds: one launch for two, no scratch.  The
// same minima, maxima and per-element arithmetic as the passes above, so the same
// bytes.  One word is the fast form, the line where it ends is explained at
// dql_small_wanted; four are for calls that must not take the two passes
// (dql_one_cluster_holds).
//
// The tensor is [rows, cols], written in rows of `pitch` bytes (zero from cols
// on); a flat tensor is one row of pitch == cols.  rowsum (may be null) gets
// the sums of the quantized rows.
constexpr int kSmallThreads = 1024;
constexpr int kSmallMaxCluster = 16;
constexpr int kSmallMaxWords = 4; // per thread

struct SmallDql {
  const float *x;
  uint8_t *y;
  int32_t *rowsum;
  float *y_scale;
  uint8_t *y_zp;
  int rows, cols, pitch;
  int row_words; // words per row: ceil(pitch / 4)
  int words;     // rows * row_words
  int vec_in;    // every whole word of x takes a 16-byte load
  int vec_out;   // every whole word of y takes a 4-byte store
  int mode;
};

template <int kWords>
__global__ void __launch_bounds__(kSmallThreads) dql_small_kernel(SmallDql p) {
  __shared__ float s_lo[kSmallThreads / 32], s_hi[kSmallThreads / 32];
  __shared__ float c_lo[kSmallMaxCluster], c_hi[kSmallMaxCluster];
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned ctas = cluster.num_blocks(), rank = cluster.block_rank();
  pdl_sync();
  const float *x = after_pdl(p.x);
  cluster.barrier_arrive(); // "has started": waited for before the first remote store
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tid = (int)(rank * kSmallThreads + threadIdx.x);
  const int nthreads = (int)(ctas * kSmallThreads);
  if (p.rowsum)
    for (int i = tid; i < p.rows; i += nthreads)
      p.rowsum[i] = 0;
  // Zeros that stand for no element change neither scalar: the range is
  // widened to hold 0 before anything is derived from it.
  float4 v[kWords];
  int row[kWords], col[kWords], have[kWords];
#pragma unroll
  for (int u = 0; u < kWords; ++u) {
    const int w = tid + u * nthreads;
    const bool in = w < p.words;
    row[u] = in ? w / p.row_words : p.rows - 1;
    col[u] = 4 * (w - row[u] * p.row_words);
    have[u] = in ? p.cols - col[u] : 0;
    v[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float *src = x + (int64_t)row[u] * p.cols + col[u];
    if (have[u] >= 4 && p.vec_in) {
      v[u] = __ldg(reinterpret_cast<const float4 *>(src));
    } else {
      if (have[u] > 0)
        v[u].x = __ldg(src);
      if (have[u] > 1)
        v[u].y = __ldg(src + 1);
      if (have[u] > 2)
        v[u].z = __ldg(src + 2);
      if (have[u] > 3)
        v[u].w = __ldg(src + 3);
    }
  }
  float lo = min3f(fminf(v[0].x, v[0].y), v[0].z, v[0].w);
  float hi = max3f(fmaxf(v[0].x, v[0].y), v[0].z, v[0].w);
#pragma unroll
  for (int u = 1; u < kWords; ++u) {
    lo = min3f(min3f(lo, v[u].x, v[u].y), v[u].z, v[u].w);
    hi = max3f(max3f(hi, v[u].x, v[u].y), v[u].z, v[u].w);
  }
  lo = warp_min(lo);
  hi = warp_max(hi);
  if (lane == 0) {
    s_lo[warp] = lo;
    s_hi[warp] = hi;
  }
  __syncthreads();
  cluster.barrier_wait();
  if (warp == 0) {
    static_assert(kSmallThreads / 32 == 32, "one value per lane");
    lo = warp_min(s_lo[lane]);
    hi = warp_max(s_hi[lane]);
    if (lane < (int)ctas) { // lane i tells CTA i
      *cluster.map_shared_rank(&c_lo[rank], lane) = lo;
      *cluster.map_shared_rank(&c_hi[rank], lane) = hi;
    }
  }
  cluster.sync(); // orders the remote stores, the zeroes in rowsum, and all loads before all stores
  lo = c_lo[0];
  hi = c_hi[0];
  for (unsigned i = 1; i < ctas; ++i) {
    lo = fminf(lo, c_lo[i]);
    hi = fmaxf(hi, c_hi[i]);
  }
  float scale, zp_f;
  dql_params_from_range(lo, hi, &scale, &zp_f, p.mode);
  if (tid == 0)
    QuantOutputs{nullptr, p.y_scale, p.y_zp}.publish(scale, zp_f);
  if (tid - lane >= p.words)
    return; // the whole warp is past the end
  const QuantConsts qc = make_quant_consts<false>(scale, zp_f, p.mode);
#pragma unroll
  for (int u = 0; u < kWords; ++u) {
    if (tid + u * nthreads - lane >= p.words)
      break;
    const bool in = tid + u * nthreads < p.words;
    const int r = row[u], c = col[u];
    uint32_t q = have[u] > 0 ? quantize_four<false>(v[u], qc) : 0u;
    if (have[u] < 4)
      q = have[u] > 0 ? q & ((1u << (8 * have[u])) - 1u) : 0u;
    if (in) {
      uint8_t *dst = p.y + (int64_t)r * p.pitch + c;
      if (p.vec_out && c + 4 <= p.pitch) {
        *reinterpret_cast<uint32_t *>(dst) = q;
      } else {
        for (int e = 0; e < 4 && c + e < p.pitch; ++e)
          dst[e] = (uint8_t)(q >> (8 * e));
      }
    }
    if (p.rowsum) {
      int32_t sum = add_bytes<false>(q, 0);
      // rows grow with the lane: first and last alike means one row
      if (__shfl_sync(0xffffffffu, r, 0) == __shfl_sync(0xffffffffu, r, 31)) {
        sum = __reduce_add_sync(0xffffffffu, sum);
        if (lane == 0)
          atomicAdd(p.rowsum + r, sum);
      } else if (in) {
        atomicAdd(p.rowsum + r, sum);
      }
    }
  }
}

// y = (x - zp) * scale, bound by HBM.  Four values a lane, so that a warp stores
// whole 512-byte lines (one value a lane: 128 bytes from 32 loads of one byte),
// and runs of kDequantUnroll * 256 such groups per block:
// 8191 x 3073 values of 8 bits 31.4 -> 20.7 us (6.1 TB/s), of 32 bits 37.5 -> 32.3.
constexpr int kDequantUnroll = 4;

// Values i .. i + 3 of x as floats, i a multiple of 4.
__device__ __forceinline__ float4 load_four(const uint8_t *x, int64_t i) {
  const uint32_t w = __ldcs(reinterpret_cast<const uint32_t *>(x + i));
  return make_float4((float)(w & 0xffu), (float)((w >> 8) & 0xffu),
      (float)((w >> 16) & 0xffu), (float)(w >> 24));
}
__device__ __forceinline__ float4 load_four(const int8_t *x, int64_t i) {
  const uint32_t w = __ldcs(reinterpret_cast<const uint32_t *>(x + i));
  return make_float4((float)(int8_t)(w & 0xffu), (float)(int8_t)((w >> 8) & 0xffu),
      (float)(int8_t)((w >> 16) & 0xffu), (float)(int8_t)(w >> 24));
}
__device__ __forceinline__ float4 load_four(const int32_t *x, int64_t i) {
  const int4 w = __ldcs(reinterpret_cast<const int4 *>(x + i));
  return make_float4((float)w.x, (float)w.y, (float)w.z, (float)w.w);
}

template <typename T>
__global__ void __launch_bounds__(256)
    dequantize_kernel(const T *__restrict__ x, int64_t n,
        const float *__restrict__ scale, const T *__restrict__ zp,
        float *__restrict__ y) {
  pdl_sync();
  x = after_pdl(x);
  scale = after_pdl(scale);
  zp = after_pdl(zp);
  const float s = __ldg(scale);
  // (subtracting +0 where there is no zero point changes no bit: a converted
  // integer is never -0)
  const float zf = zp ? (float)*zp : 0.0f;
  const int64_t n4 = n >> 2;
  float4 *y4 = reinterpret_cast<float4 *>(y);
  constexpr int kRun = kDequantUnroll * 256;
  for (int64_t base = (int64_t)blockIdx.x * kRun + threadIdx.x; base < n4;
       base += (int64_t)gridDim.x * kRun) {
    float4 v[kDequantUnroll];
#pragma unroll
    for (int u = 0; u < kDequantUnroll; ++u)
      if (base + u * 256 < n4)
        v[u] = load_four(x, 4 * (base + u * 256));
#pragma unroll
    for (int u = 0; u < kDequantUnroll; ++u)
      if (base + u * 256 < n4)
        y4[base + u * 256] = make_float4(__fmul_rn(__fsub_rn(v[u].x, zf), s),
            __fmul_rn(__fsub_rn(v[u].y, zf), s), __fmul_rn(__fsub_rn(v[u].z, zf), s),
            __fmul_rn(__fsub_rn(v[u].w, zf), s));
  }
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
    const int64_t i = (n4 << 2) + threadIdx.x;
    y[i] = __fmul_rn(__fsub_rn((float)x[i], zf), s);
  }
}

// The same one value at a time, for tensors that do not start on a whole group of
// four.  A loop of its own over a grid of its own (8 blocks per SM at most): as a
// remainder of the kernel above, on its grid, 30 M values of 8 bits took 70 us,
// of 32 bits 89; so 38 and 44 (20 000 values 6.2 and 4.1).
template <typename T>
__global__ void __launch_bounds__(256)
    dequantize_single_kernel(const T *__restrict__ x, int64_t n,
        const float *__restrict__ scale, const T *__restrict__ zp,
        float *__restrict__ y) {
  pdl_sync();
  x = after_pdl(x);
  scale = after_pdl(scale);
  zp = after_pdl(zp);
  const float s = __ldg(scale);
  const float zf = zp ? (float)*zp : 0.0f;
  const bool has_zp = zp != nullptr;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float xf = (float)x[i];
    y[i] = __fmul_rn(has_zp ? __fsub_rn(xf, zf) : xf, s);
  }
}

static int grid_for(int64_t work_items, int per_block) {
  int64_t want = ceil_div(work_items, per_block);
  const int64_t cap = (int64_t)sm_count() * 8;
  if (want < 1)
    want = 1;
  return (int)(want < cap ? want : cap);
}

// Blocks of the passes that write one value per value.  What comes from L2 is
// fastest with the blocks that are resident at once (16 Mi values: 13.0 us, with
// a short block per run 15.8); what comes from HBM with short blocks, up to 64 per
// SM, of which the last round is a small part (64 Mi: 51.6, resident ones 54.6).
static int pass_grid(int64_t n, int run, int resident) { // blocks per SM, 0: not only those
  int64_t want = ceil_div(n, run);
  const int64_t cap = (int64_t)sm_count() * (resident ? resident : 64);
  if (want < 1)
    want = 1;
  return (int)(want < cap ? want : cap);
}

// float4 per thread and run of the quantize pass: four, fewer while that would
// leave SMs without a block.
static int quant_unroll(int64_t n) {
  const int64_t per = ceil_div(n, (int64_t)sm_count() * 2 * kDqlThreads * 4);
  return (int)(per < 1 ? 1 : per < kQuantUnroll ? per : kQuantUnroll);
}

// Whether quantize_wide_kernel takes a pass.  Behind a producer (an encoder's) from 24000
// values: its few blocks leave the GEMM behind it the SMs (2 x 128 tokens of 768 567 -> 544 us,
// 33 tokens 410 -> 405, but 16 tokens 431 -> 449); else where a block per 4096 values no longer
// leaves SMs idle (given scale: 230000 values 1.95 -> 1.84 us, 187392 1.89 and 2.00).
static bool quant_wide(const float *x, int64_t n, const uint8_t *y, bool behind_producer) {
  return ((uintptr_t)x & 31u) == 0 && ((uintptr_t)y & 7u) == 0 &&
         n >= (behind_producer ? 24000 : 200000);
}

template <typename T>
static void launch_dequantize(const T *x, int64_t n, const float *scale, const T *zp,
    float *y, cudaStream_t st) {
  const bool whole = ((uintptr_t)x & (4 * sizeof(T) - 1)) == 0 && ((uintptr_t)y & 15u) == 0;
  // Set up behind its predecessor whatever the size, as the quantize pass with a given
  // scale is: without shared memory and with few registers its blocks
  // take nothing that one needs.  2 us of each call, 1 Mi values 4.2 -> 2.1, 8191 x 3073 of 8
  // bits 22.7 -> 20.7, 64 Mi 55.0 -> 52.3.
  if (whole)
    (void)launch_pdl(dequantize_kernel<T>, pass_grid(n, 256 * 4 * kDequantUnroll, 0), 256, 0,
        st, 0, true, x, n, scale, zp, y);
  else
    (void)launch_pdl(
        dequantize_single_kernel<T>, grid_for(n, 256 * 4), 256, 0, st, 0, true, x, n, scale, zp, y);
}

namespace {

template <bool kSigned>
int launch_quantize_pass(const float *x, int64_t n, uint8_t *y, const QuantSource &src,
    const QuantOutputs &outs, cudaStream_t st) {
  const int unroll = quant_unroll(n);
  // Behind the reduction: resident blocks, for each block folds all partials, and
  // set up while it runs, whatever the size (it holds no shared memory that
  // matters; 64 Mi values 115 us with short blocks, 106 with resident ones, 103
  // with the overlap).
  const bool folds = src.parts.count > 0;
  // (what a producer on the device has just left lies in L2 up to some 100 MB; a
  // caller's own tensor may come from anywhere)
  const bool in_l2 = src.range && n <= ((int64_t)24 << 20);
  // (a given scale: 64 Mi values 55.2 -> 52.8 us; a pass of an encoder's, between GEMMs, by
  // the rule)
  const bool overlap = folds || src.scale || pdl_pays(n);
  // What a reduction or a producer has just had: what L2 still holds of it survives
  // until the pass gets there if what the pass has read may go first (the whole call, 16 Mi
  // values 25.9 and so 24.0 us, 32 Mi 50.8 and 45.4; encoder large 64 x 512 24.8 and 24.6 ms,
  // 4 x 512 2418 and 2426 us).  Beyond what L2 could hold of it plain loads are faster (128 Mi 187
  // and 194), as for a given scale (64 Mi 49.0 and 51.4).
  const bool once = !src.scale && n <= ((int64_t)96 << 20);
  // Few values behind a reduction: two blocks per SM.  It still holds SMs when this is set up,
  // and of more blocks some start a round late (3.6 M values 9.3 us with four, 7.7 with two, 5 M
  // 9.7 and 12.5; between the kernels of an encoder four are better at any size).
  const int resident = folds && n <= 4800000 ? 2 : folds || in_l2 ? kWideBlocksPerSm : 0;
  if (quant_wide(x, n, y, src.range != nullptr)) {
    const auto kernel =
        !kSigned && once ? quantize_wide_kernel<kSigned, !kSigned> : quantize_wide_kernel<kSigned, false>;
    const int grid = pass_grid(n, kWideGroups * 8 * kDqlThreads, resident);
    // Two or three blocks per SM, kept apart (encoder base 8 x 128 716 -> 708 us, 3 x 500 1122 ->
    // 1107, large 2 x 512 1850 -> 1823; one per SM is better left to the GEMM behind it, 2 x 128 515
    // and 518).
    const int64_t per_sm = ceil_div((int64_t)grid, (int64_t)sm_count());
    size_t spread = 0;
    if (src.range && overlap && per_sm > 1 && per_sm < kWideBlocksPerSm) {
      static PerDeviceInt can[2]; // 1: yes, 2: no
      PerDeviceInt &c = can[once];
      if (!c.get()) {
        c.set(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                  (int)spread_bytes(2)) == cudaSuccess
                  ? 1
                  : 2);
        (void)cudaGetLastError();
      }
      spread = c.get() == 1 ? spread_bytes(per_sm) : 0;
    }
    OMCUDA_CHECK(launch_pdl(kernel, (unsigned)grid, kDqlThreads, spread, st, 0, overlap, x, n, y,
        src, outs, quant_mode()));
  } else if (((uintptr_t)x & 15u) == 0 && ((uintptr_t)y & 3u) == 0)
    OMCUDA_CHECK(launch_pdl(quantize_kernel<kSigned>,
        pass_grid(n, kDqlThreads * 4 * unroll, folds || in_l2 ? 8 : 0), kDqlThreads, 0, st, 0,
        overlap, x, n, y, src, outs, quant_mode(), unroll));
  else
    OMCUDA_CHECK(launch_pdl(quantize_single_kernel<kSigned>, grid_for(n, kDqlThreads * 4),
        kDqlThreads, 0, st, 0, overlap, x, n, y, src, outs, quant_mode()));
  OMCUDA_CHECK_LAUNCH("quantize_kernel");
  return OMCUDA_OK;
}

// DynamicQuantizeLinear's reduction alone.  roomy: the pass behind can wait for the registers of
// deep blocks (see `deep`).
int launch_range_parts(const float *x, int64_t n, void *scratch, RangeParts *parts,
    cudaStream_t st, bool overlap, bool roomy = true, int32_t *sums = nullptr, int zeros = 0) {
  float2 *part = scratch_parts(scratch);
  // Runs of one to eight float4 a thread, so that about a third of the SMs has a
  // block until those are full: no block without work, whose empty partial every
  // block behind would fold.  1 Mi values (the whole call) 7.7 -> 5.3 us, 524288 5.7 ->
  // 5.1, 98304 4.5 -> 4.3 against runs of eight and a block per 2048 values, most of
  // them empty.  With a block per SM the call alone gains as much (5.2), but what is
  // set up behind loses: linear 777 x 1001 x 1537 20.3 so, 19.4 with one per SM, 18.7.
  const int64_t per = ceil_div(n, (int64_t)(sm_count() / 3) * kRangeThreads * 4);
  const int unroll = (int)(per < 1 ? 1 : per < kRangeUnroll ? per : kRangeUnroll);
  const bool aligned = ((uintptr_t)x & 15u) == 0; // (else four single values a thread)
  int64_t grid = ceil_div(n, (int64_t)kRangeThreads * 4 * (aligned ? unroll : 1));
  const int64_t cap = (int64_t)sm_count() * kRangeBlocksPerSm;
  grid = grid < 1 ? 1 : grid < cap ? grid : cap;
  if (grid > kRangeMaxParts)
    grid = kRangeMaxParts;
  const bool full = unroll == kRangeUnroll;
  // Small blocks, one float4 a thread, while they are few enough to be folded: the fewer
  // warps an SM has, the sooner each is through.  What the device takes for the whole call
  // (a caller's host may take longer: some 10 us for a linear through the Python binding):
  // 70000 values 4.21 -> 3.96 us, 100000 4.23 -> 4.06, linear 128 x 768 x 768 8.71 -> 8.59, 35 x
  // 2500 x 640 9.42 -> 9.08, but 100 x 1024 x 1024 9.16 and 9.25; 150000 4.32 and 4.49.
  const int64_t small_blocks = ceil_div(n, (int64_t)kRangeFewThreads * 4);
  const bool few = aligned && 2 * small_blocks <= 3 * sm_count();
  if (few)
    grid = small_blocks < 1 ? 1 : small_blocks;
  // All loads of a run in flight, except where the blocks are one to two per SM: more of
  // them than fit with those registers beside what else is resident (3.1 M values 6.8 us
  // without, 8.3 with; 6 M 11.9 and 10.8).
  const bool deep = (roomy && grid <= sm_count()) || grid > 2 * sm_count();
  const auto kernel =
      few     ? (sums ? dql_minmax_kernel<false, true, kRangeFewThreads, true>
                      : dql_minmax_kernel<false, false, kRangeFewThreads, true>)
      : !full ? (sums ? dql_minmax_kernel<false, true, kRangeThreads, true>
                      : dql_minmax_kernel<false, false, kRangeThreads, true>)
      : deep  ? (sums ? dql_minmax_kernel<true, true, kRangeThreads, true>
                      : dql_minmax_kernel<true, false, kRangeThreads, true>)
              : (sums ? dql_minmax_kernel<true, true, kRangeThreads, false>
                      : dql_minmax_kernel<true, false, kRangeThreads, false>);
  OMCUDA_CHECK(launch_pdl(kernel, (unsigned)grid, few ? kRangeFewThreads : kRangeThreads, 0, st, 0,
      overlap, x, n, part, few ? 1 : unroll, sums, zeros));
  OMCUDA_CHECK_LAUNCH("dql_minmax_kernel");
  parts->part = part;
  parts->count = (int)grid;
  return OMCUDA_OK;
}

} // namespace

int launch_dql_rows(const float *x, int64_t rows, int64_t cols, int64_t pitch, uint8_t *y,
    int32_t *rowsum, float *y_scale, uint8_t *y_zp, void *scratch, cudaStream_t st) {
  const bool warps = rows >= (int64_t)sm_count() * 4;
  // Few rows, long ones: about one block per SM, but none with less than the four
  // words a thread keeps in flight.  u8 weights, N = 256: 1 x 100000 40 -> 21 us, 8 x
  // 14336 19.8 -> 18.6, 16 x 14336 21.2 -> 19.8; two per SM cost 128 x 8192 0.5.
  int64_t split = 1;
  if (rows > 0 && rows < sm_count() && pitch < (int64_t)1 << 30) { // (32-bit columns)
    const int64_t most = ceil_div(pitch, kRowsUnroll * 4 * kDqlThreads);
    split = sm_count() / rows;
    split = split < most ? split : most > 0 ? most : 1;
  }
  RangeParts parts;
  const int64_t blocks = warps ? ceil_div(rows, kDqlThreads / 32) : rows * split;
  const int vec_in = ((uintptr_t)x & 15u) == 0 && cols % 4 == 0;
  // The reduction's blocks take half the registers of an SM if deep, which pays but in front of
  // long rows that a warp each takes value by value: those take longest and want to be in
  // place.  Linears, deep and not: 900 x 1001 x 768 13.0 and 12.4 us, 777 x 1385 x 1024 14.6 and 13.9, 650 x
  // 3001 x 1024 20.0 and 18.6, 1544 x 1385 x 768 17.5 and 16.6, but of shorter rows 1500 x 501 x 3072 14.5
  // and 15.5, 1200 x 801 x 1024 13.8 and 14.1, with four values a load 1544 x 768 x 3072 18.4 and 19.6, 700 x
  // 1536 x 1024 13.8 and 14.2, a block per row 147 x 9001 x 2048 21.6 and 23.0, 300 x 4800 x 1600 16.5 and 17.1.
  const bool roomy = !(warps && !vec_in && cols >= 1000);
  int rc = launch_range_parts(x, rows * cols, scratch, &parts, st, pdl_pays(rows * cols),
      roomy, split > 1 ? rowsum : nullptr, (int)rows);
  if (rc != OMCUDA_OK)
    return rc;
  const int64_t cap = (int64_t)sm_count() * 8;
  OMCUDA_CHECK(launch_pdl(warps       ? quantize_rows_kernel<1, false>
                          : split > 1 ? quantize_rows_kernel<8, true>
                                      : quantize_rows_kernel<8, false>,
      (unsigned)(blocks < cap ? blocks : cap), kDqlThreads, 0, st, 0, pdl_pays(rows * cols), x,
      rows, (int)cols, (int)pitch, y, rowsum, parts, QuantOutputs{nullptr, y_scale, y_zp},
      vec_in, (int)split, quant_mode()));
  OMCUDA_CHECK_LAUNCH("quantize_rows_kernel");
  return OMCUDA_OK;
}

namespace {

// The largest cluster of dql_small_kernel the device can place.
int small_cluster_limit() {
  static PerDeviceInt limit;
  int n = limit.get();
  if (n == 0) {
    n = 8; // always placeable
    cudaLaunchConfig_t q = {};
    q.gridDim = dim3(kSmallMaxCluster, 1, 1);
    q.blockDim = dim3(kSmallThreads, 1, 1);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kSmallMaxCluster;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    q.attrs = at;
    q.numAttrs = 1;
    int a = 0, b = 0;
    if (cudaFuncSetAttribute(dql_small_kernel<1>,
            cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaFuncSetAttribute(dql_small_kernel<kSmallMaxWords>,
            cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&a, dql_small_kernel<1>, &q) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&b, dql_small_kernel<kSmallMaxWords>, &q) ==
            cudaSuccess &&
        a > 0 && b > 0)
      n = kSmallMaxCluster;
    (void)cudaGetLastError();
    limit.set(n);
  }
  return n;
}

} // namespace

bool dql_small_wanted(int64_t rows, int64_t pitch) {
  // One word a thread, 65536 values in 16 CTAs: 8192 values 3.5 us, 32768 3.6, where
  // two launches take 4.4 at any size up to 200 000.  With more words a thread the
  // few SMs of one cluster lose to the whole machine: two, 131072 values, 5.0 us.
  const int64_t words = (int64_t)kSmallThreads * small_cluster_limit();
  return rows <= words && pitch <= 4 * words && rows * ceil_div(pitch, 4) <= words;
}

bool dql_one_cluster_holds(int64_t n) {
  return n <= (int64_t)4 * kSmallMaxWords * kSmallThreads * small_cluster_limit();
}

bool dql_in_place(const float *x, int64_t n, const uint8_t *y, const float *y_scale,
    const uint8_t *y_zp) {
  const int64_t bytes = n * (int64_t)sizeof(float);
  return ranges_overlap(x, bytes, y, n) || ranges_overlap(x, bytes, y_scale, sizeof(float)) ||
         ranges_overlap(x, bytes, y_zp, 1);
}

int launch_dql_small(const float *x, int64_t rows, int64_t cols, int64_t pitch,
    uint8_t *y, int32_t *rowsum, float *y_scale, uint8_t *y_zp, cudaStream_t st) {
  SmallDql p;
  p.x = x;
  p.y = y;
  p.rowsum = rowsum;
  p.y_scale = y_scale;
  p.y_zp = y_zp;
  p.rows = (int)rows;
  p.cols = (int)cols;
  p.pitch = (int)pitch;
  p.row_words = (int)ceil_div(pitch, 4);
  p.words = (int)(rows * p.row_words);
  p.vec_in = ((uintptr_t)x & 15u) == 0 && (rows == 1 || cols % 4 == 0);
  p.vec_out = ((uintptr_t)y & 3u) == 0 && (rows == 1 || pitch % 4 == 0);
  p.mode = quant_mode();
  unsigned ctas = 1;
  while (ctas * kSmallThreads < (unsigned)p.words && ctas < (unsigned)small_cluster_limit())
    ctas *= 2;
  OMCUDA_CHECK(launch_pdl((unsigned)p.words <= ctas * kSmallThreads
                              ? dql_small_kernel<1>
                              : dql_small_kernel<kSmallMaxWords>,
      ctas, kSmallThreads, 0, st, ctas, true, p));
  count_launch();
  return OMCUDA_OK;
}

} // namespace omcuda

using namespace omcuda;

extern "C" int64_t omcudaDevDqlScratchBytes(int64_t) {
  return kScratchBytes;
}

int omcuda::launch_dql(const float *x, int64_t n, uint8_t *y, float *y_scale, uint8_t *y_zp,
    void *scratch, cudaStream_t st, bool alone) {
  if (n < 0 || (n > 0 && (!x || !y)) || !scratch)
    return fail(OMCUDA_EINVAL, "DynamicQuantizeLinear: bad argument");
  if (dql_small_wanted(1, n) ||
      (dql_one_cluster_holds(n) && dql_in_place(x, n, y, y_scale, y_zp)))
    return launch_dql_small(x, 1, n, n, y, nullptr, y_scale, y_zp, st);
  RangeParts parts;
  // Set up early whatever the size where what runs before is as a rule a pass like this
  // (64 Mi values 100.7 -> 99.0 us), but not behind a GEMM of a long linear, whose SMs its
  // blocks would take (8192 x 4096 x 4096 149 and 155).
  int rc = launch_range_parts(x, n, scratch, &parts, st, alone || pdl_pays(n));
  if (rc != OMCUDA_OK)
    return rc;
  return launch_quantize_pass<false>(x, n, y, QuantSource{parts, nullptr, nullptr, nullptr},
      QuantOutputs{nullptr, y_scale, y_zp}, st);
}

extern "C" int omcudaDevDynamicQuantizeLinear(const float *x, int64_t n,
    uint8_t *y, float *y_scale, uint8_t *y_zp, void *scratch, void *stream) {
  return launch_dql(x, n, y, y_scale, y_zp, scratch, (cudaStream_t)stream, false);
}

extern "C" int omcudaDevRangeFold(const float *x, int64_t n, void *range, void *stream) {
  if (n < 0 || (n > 0 && !x) || !range)
    return fail(OMCUDA_EINVAL, "RangeFold: bad argument");
  if (n == 0)
    return OMCUDA_OK;
  int grid = grid_for(n, kDqlThreads * 16);
  range_fold_kernel<<<grid, kDqlThreads, 0, (cudaStream_t)stream>>>(x, n, (uint32_t *)range);
  OMCUDA_CHECK_LAUNCH("range_fold_kernel");
  return OMCUDA_OK;
}

extern "C" int omcudaDevQuantizeFromRange(const float *x, int64_t n, void *range,
    uint8_t *y, float *params, float *y_scale, uint8_t *y_zp, void *stream) {
  if (n < 0 || (n > 0 && (!x || !y)) || !range || !params)
    return fail(OMCUDA_EINVAL, "QuantizeFromRange: bad argument");
  cudaStream_t st = (cudaStream_t)stream;
  // One launch: every block derives the scalars from the range itself (a
  // block of its own when there is nothing to quantize).
  return launch_quantize_pass<false>(x, n, y,
      QuantSource{RangeParts{nullptr, 0}, (const uint32_t *)range, nullptr, nullptr},
      QuantOutputs{params, y_scale, y_zp}, st);
}

extern "C" int omcudaDevQuantizeLinear(const float *x, int64_t n, void *y,
    int y_signed, const float *scale, const void *zp, void *stream) {
  if (n < 0 || (n > 0 && (!x || !y)) || !scale)
    return fail(OMCUDA_EINVAL, "QuantizeLinear: bad argument");
  if (n == 0)
    return OMCUDA_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const QuantSource src{RangeParts{nullptr, 0}, nullptr, scale, zp};
  return y_signed ? launch_quantize_pass<true>(x, n, (uint8_t *)y, src, QuantOutputs{}, st)
                  : launch_quantize_pass<false>(x, n, (uint8_t *)y, src, QuantOutputs{}, st);
}

extern "C" int omcudaDevDequantizeLinear(const void *x, int dtype, int64_t n,
    const float *scale, const void *zp, float *y, void *stream) {
  if (n < 0 || (n > 0 && (!x || !y)) || !scale || dtype < 0 || dtype > 2)
    return fail(OMCUDA_EINVAL, "DequantizeLinear: bad argument");
  if (n == 0)
    return OMCUDA_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (quant_mode() & OMCUDA_MODE_NO_ZERO_POINT)
    zp = nullptr; // the reference drops the subtraction (Math/Elementwise.cpp:1453)
  if (dtype == 0)
    launch_dequantize((const uint8_t *)x, n, scale, (const uint8_t *)zp, y, st);
  else if (dtype == 1)
    launch_dequantize((const int8_t *)x, n, scale, (const int8_t *)zp, y, st);
  else
    launch_dequantize((const int32_t *)x, n, scale, (const int32_t *)zp, y, st);
  OMCUDA_CHECK_LAUNCH("dequantize_kernel");
  return OMCUDA_OK;
}
