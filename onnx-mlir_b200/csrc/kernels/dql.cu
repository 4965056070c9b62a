// DynamicQuantizeLinear / QuantizeLinear / DequantizeLinear kernels.
//
// Semantics follow onnx-mlir's lowering:
//   min/max   src/Conversion/ONNXToKrnl/Math/Reduction.cpp:394-548 (minnum/maxnum,
//             identities +inf/-inf)
//   params    src/Conversion/ONNXToKrnl/Quantization/DynamicQuantizeLinear.cpp:43-84
//   quantize  src/Conversion/ONNXToKrnl/Quantization/QuantizeLinear.cpp:122-145
//   dequant   src/Conversion/ONNXToKrnl/Math/Elementwise.cpp:1438-1461
//
// Layout: tensors are flat, dense, row-major.  The reduction runs as a
// single-pass grid reduction: every block leaves its partial min/max in
// scratch, takes a ticket, and the block that draws the last ticket folds the
// partials and derives scale and zero point, so no block ever waits on
// another.  The quantize pass is a second launch that reads the two scalars
// from device memory; for tensors that fit in L2 its read of x is served from
// there.
#include <cooperative_groups.h>

#include "../common.cuh"
#include "../runtime/internal.h"
#include "quantize.cuh"

namespace cg = cooperative_groups;

namespace omcuda {

static constexpr int kDqlThreads = 256;
static constexpr int kDqlMaxBlocks = 2048;
static constexpr int kQuantUnroll = 4;

struct DqlScratch {
  unsigned int ticket;
  unsigned int pad[15];
  float part_min[kDqlMaxBlocks];
  float part_max[kDqlMaxBlocks];
  float params[4]; // scale, zero point as float
};

__global__ void __launch_bounds__(kDqlThreads)
    dql_minmax_kernel(const float *__restrict__ x, int64_t n,
        DqlScratch *__restrict__ scr, float *__restrict__ y_scale,
        uint8_t *__restrict__ y_zp, int mode) {
  pdl_sync();
  x = after_pdl(x);
  float lo = INFINITY, hi = -INFINITY;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  const bool aligned = ((uintptr_t)x & 15u) == 0;
  if (aligned) {
    const int64_t n4 = n >> 2;
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    // Eight independent 16-byte loads in flight per thread per trip: with all
    // 2048 threads of an SM resident that is 256 KiB outstanding per SM, well
    // above what HBM latency times bandwidth asks for.
    int64_t i = tid;
    for (; i + 7 * nthreads < n4; i += 8 * nthreads) {
      float4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        v[u] = __ldcs(x4 + i + u * nthreads);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        lo = fminf(lo, fminf(fminf(v[u].x, v[u].y), fminf(v[u].z, v[u].w)));
        hi = fmaxf(hi, fmaxf(fmaxf(v[u].x, v[u].y), fmaxf(v[u].z, v[u].w)));
      }
    }
    for (; i < n4; i += nthreads) {
      float4 a = __ldcs(x4 + i);
      lo = fminf(lo, fminf(fminf(a.x, a.y), fminf(a.z, a.w)));
      hi = fmaxf(hi, fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)));
    }
    for (int64_t j = (n4 << 2) + tid; j < n; j += nthreads) {
      float v = __ldg(x + j);
      lo = fminf(lo, v);
      hi = fmaxf(hi, v);
    }
  } else {
    for (int64_t j = tid; j < n; j += nthreads) {
      float v = __ldg(x + j);
      lo = fminf(lo, v);
      hi = fmaxf(hi, v);
    }
  }
  lo = warp_min(lo);
  hi = warp_max(hi);
  __shared__ float s_lo[kDqlThreads / 32], s_hi[kDqlThreads / 32];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    s_lo[warp] = lo;
    s_hi[warp] = hi;
  }
  __syncthreads();
  if (warp == 0) {
    lo = lane < kDqlThreads / 32 ? s_lo[lane] : INFINITY;
    hi = lane < kDqlThreads / 32 ? s_hi[lane] : -INFINITY;
    lo = warp_min(lo);
    hi = warp_max(hi);
    if (lane == 0) {
      scr->part_min[blockIdx.x] = lo;
      scr->part_max[blockIdx.x] = hi;
      __threadfence();
      unsigned int t = atomicAdd(&scr->ticket, 1u);
      s_last = (t == gridDim.x - 1);
    }
  }
  __syncthreads();
  if (!s_last)
    return;
  // Last block: fold the partials (order does not matter for min/max).
  __threadfence();
  lo = INFINITY;
  hi = -INFINITY;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
    lo = fminf(lo, __ldcg(&scr->part_min[i]));
    hi = fmaxf(hi, __ldcg(&scr->part_max[i]));
  }
  lo = warp_min(lo);
  hi = warp_max(hi);
  __syncthreads();
  if (lane == 0) {
    s_lo[warp] = lo;
    s_hi[warp] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kDqlThreads / 32; ++w) {
      lo = fminf(lo, s_lo[w]);
      hi = fmaxf(hi, s_hi[w]);
    }
    float s, z;
    dql_params_from_range(lo, hi, &s, &z, mode);
    scr->params[0] = s;
    scr->params[1] = z;
    if (y_scale)
      *y_scale = s;
    if (y_zp)
      *y_zp = (uint8_t)(unsigned int)z; // fptoui then trunc; z is in [0,255]
    scr->ticket = 0; // leave the scratch ready for the next call
  }
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

// Where the range-driven form of the kernel leaves its scalars.
struct QuantOutputs {
  float *params;  // {scale, zero point as float}
  float *y_scale; // the op's y_scale output, may be null
  uint8_t *y_zp;  // the op's y_zero_point output, may be null
};

// params: {scale, zp as float}.  If zp8 is non-NULL the zero point is read
// from it instead (QuantizeLinear with a given 8-bit zero point).  If range is
// non-NULL, scale and zero point are derived from that running {min,max}
// (ordered-uint encoding, see f32_to_ordered) as DynamicQuantizeLinear does.
template <bool kSigned>
__global__ void __launch_bounds__(kDqlThreads)
    quantize_kernel(const float *__restrict__ x, int64_t n,
        uint8_t *__restrict__ y, const float *__restrict__ params,
        const float *__restrict__ scale_ptr, const void *__restrict__ zp8,
        int has_zp, const uint32_t *__restrict__ range, QuantOutputs outs, int mode,
        int unroll) {
  pdl_sync();
  x = after_pdl(x);
  params = after_pdl(params);
  scale_ptr = after_pdl(scale_ptr);
  zp8 = after_pdl(zp8);
  range = after_pdl(range);
  // A block takes runs of unroll * 256 neighbouring float4 (16 KiB at most), the
  // loads of the first before it derives the scalars: three dependent divides
  // that a launch on a small tensor would otherwise spend before it asks for data.
  // Runs and not a stride of the whole grid, and only four loads in flight per
  // thread so that more blocks fit: 64 Mi values 67.0 -> 64.1 us, an encoder run of
  // 1 x 61 resident tokens 741 -> 659 us, of 32 x 128 1903 -> 1839.
  const bool aligned = (((uintptr_t)x & 15u) == 0) && (((uintptr_t)y & 3u) == 0);
  const int64_t n4 = aligned ? n >> 2 : 0;
  const float4 *x4 = reinterpret_cast<const float4 *>(x);
  uint32_t *y4 = reinterpret_cast<uint32_t *>(y);
  const int run = unroll * kDqlThreads;
  int64_t base = (int64_t)blockIdx.x * run + threadIdx.x;
  float4 v[kQuantUnroll];
#pragma unroll
  for (int u = 0; u < kQuantUnroll; ++u)
    if (u < unroll && base + u * kDqlThreads < n4)
      v[u] = __ldcs(x4 + base + u * kDqlThreads);
  float scale, zp_f;
  if (range) {
    // Scale and zero point straight from a producer's running range (every
    // thread derives the same two scalars; block 0 also publishes them for
    // the ops that follow).
    dql_params_from_range(ordered_to_f32(__ldg(range)), ordered_to_f32(__ldg(range + 1)),
        &scale, &zp_f, mode);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      outs.params[0] = scale;
      outs.params[1] = zp_f;
      if (outs.y_scale)
        *outs.y_scale = scale;
      if (outs.y_zp)
        *outs.y_zp = (uint8_t)(unsigned int)zp_f; // fptoui; zp_f is in [0,255]
    }
  } else if (params) {
    scale = __ldg(params);
    zp_f = __ldg(params + 1);
  } else {
    scale = __ldg(scale_ptr);
    if (!has_zp)
      zp_f = 0.0f;
    else if (kSigned)
      zp_f = (float)*reinterpret_cast<const int8_t *>(zp8);
    else
      zp_f = (float)*reinterpret_cast<const uint8_t *>(zp8);
  }
  const QuantConsts qc = make_quant_consts<kSigned>(scale, zp_f, mode);
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
  // what is left of a word, or everything when the addresses are not aligned
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t j = (n4 << 2) + tid; j < n; j += nthreads)
    y[j] = (uint8_t)quantize_one<kSigned>(__ldg(x + j), qc);
}

// The quantize pass for rows whose length is no multiple of 16, written in the
// aligned rows the GEMM kernels take (zero from cols up to pitch), with the sums
// of the quantized rows where the weight has a zero point.  One block per row
// at a time: a thread makes one output word from four neighbouring values.
__global__ void __launch_bounds__(kDqlThreads)
    quantize_rows_kernel(const float *__restrict__ x, int64_t rows, int cols, int pitch,
        uint8_t *__restrict__ y, int32_t *__restrict__ rowsum,
        const float *__restrict__ params, int mode) {
  pdl_sync();
  x = after_pdl(x);
  params = after_pdl(params);
  __shared__ int32_t part[kDqlThreads / 32];
  const QuantConsts qc = make_quant_consts<false>(__ldg(params), __ldg(params + 1), mode);
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    const float *xr = x + r * cols;
    uint32_t *yr = reinterpret_cast<uint32_t *>(y + r * pitch);
    int32_t sum = 0;
    for (int j = threadIdx.x; 4 * j < pitch; j += kDqlThreads) {
      const int have = cols - 4 * j;
      float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < have)
          v[e] = __ldg(xr + 4 * j + e);
      uint32_t w = 0;
      if (have > 0)
        w = quantize_four<false>(make_float4(v[0], v[1], v[2], v[3]), qc);
      if (have > 0 && have < 4)
        w &= (1u << (8 * have)) - 1u;
      yr[j] = w;
      sum = add_bytes<false>(w, sum);
    }
    if (rowsum) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
      __syncthreads(); // part[] of the row before has been read
      if ((threadIdx.x & 31) == 0)
        part[threadIdx.x >> 5] = sum;
      __syncthreads();
      if (threadIdx.x == 0) {
        int32_t s = 0;
        for (int w = 0; w < kDqlThreads / 32; ++w)
          s += part[w];
        rowsum[r] = s;
      }
    }
  }
}

// DynamicQuantizeLinear of a tensor that one cluster can hold in registers: up
// to 16 CTAs x 1024 threads x 4 words of four values.  What bounds small
// tensors is launches (scratch memset, reduction, quantize pass: three, each
// with its own way through memory); here every thread loads its values once,
// the CTAs exchange their {min,max} through distributed shared memory, every
// thread derives the two scalars and quantizes what it still holds.  The same
// minima, maxima and per-element arithmetic as the passes above, so the same
// bytes.  The operator on 1000 values 10.3 -> 5.2 us, on 98304 12.6 -> 8.2, on
// 262144 13.3 -> 10.3; the linear 128 x 768 x 768 22.5 -> 16.9.
//
// The tensor is [rows, cols], written in rows of `pitch` bytes (zero from cols
// on); a flat tensor is one row of pitch == cols.  rowsum (may be null) gets
// the sums of the quantized rows.
constexpr int kSmallThreads = 1024;
constexpr int kSmallMaxWords = 4; // per thread
constexpr int kSmallMaxCluster = 16;

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
    for (int r = tid; r < p.rows; r += nthreads)
      p.rowsum[r] = 0;
  float4 v[kWords];
  float lo = INFINITY, hi = -INFINITY;
#pragma unroll
  for (int u = 0; u < kWords; ++u) {
    const int w = tid + u * nthreads;
    v[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (w >= p.words)
      continue;
    const int r = w / p.row_words, c = 4 * (w - r * p.row_words);
    const float *src = x + (int64_t)r * p.cols + c;
    const int have = p.cols - c;
    if (have >= 4 && p.vec_in) {
      v[u] = __ldg(reinterpret_cast<const float4 *>(src));
    } else {
      if (have > 0)
        v[u].x = __ldg(src);
      if (have > 1)
        v[u].y = __ldg(src + 1);
      if (have > 2)
        v[u].z = __ldg(src + 2);
      if (have > 3)
        v[u].w = __ldg(src + 3);
    }
  }
  // Zeros that stand for no element change neither scalar: the range is
  // widened to hold 0 before anything is derived from it.
#pragma unroll
  for (int u = 0; u < kWords; ++u) {
    lo = fminf(lo, fminf(fminf(v[u].x, v[u].y), fminf(v[u].z, v[u].w)));
    hi = fmaxf(hi, fmaxf(fmaxf(v[u].x, v[u].y), fmaxf(v[u].z, v[u].w)));
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
  cluster.sync(); // orders the remote stores, and the zeroes in rowsum
  lo = c_lo[0];
  hi = c_hi[0];
  for (unsigned i = 1; i < ctas; ++i) {
    lo = fminf(lo, c_lo[i]);
    hi = fmaxf(hi, c_hi[i]);
  }
  float scale, zp_f;
  dql_params_from_range(lo, hi, &scale, &zp_f, p.mode);
  if (tid == 0) {
    if (p.y_scale)
      *p.y_scale = scale;
    if (p.y_zp)
      *p.y_zp = (uint8_t)(unsigned int)zp_f; // fptoui; zp_f is in [0,255]
  }
  const QuantConsts qc = make_quant_consts<false>(scale, zp_f, p.mode);
#pragma unroll
  for (int u = 0; u < kWords; ++u) {
    const int w = tid + u * nthreads;
    if (w - lane >= p.words)
      break; // the whole warp is past the end
    const bool in = w < p.words;
    const int r = in ? w / p.row_words : p.rows - 1;
    const int c = 4 * (w - r * p.row_words);
    const int have = in ? p.cols - c : 0;
    uint32_t q = have > 0 ? quantize_four<false>(v[u], qc) : 0u;
    if (have < 4)
      q = have > 0 ? q & ((1u << (8 * have)) - 1u) : 0u;
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
// 8191 x 3073 values of 8 bits 31.4 -> 22.7 us (5.5 TB/s), of 32 bits 37.5 -> 35.3.
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
  int64_t cap = (int64_t)sm_count() * 8;
  if (cap > kDqlMaxBlocks)
    cap = kDqlMaxBlocks;
  if (want < 1)
    want = 1;
  return (int)(want < cap ? want : cap);
}

// Blocks of the passes that write one value per value: short ones, as many as
// there are runs (up to 64 per SM), so that the last round is a small part.
static int pass_grid(int64_t n, int run) {
  int64_t want = ceil_div(n, run);
  const int64_t cap = (int64_t)sm_count() * 64;
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

template <typename T>
static void launch_dequantize(const T *x, int64_t n, const float *scale, const T *zp,
    float *y, cudaStream_t st) {
  const bool whole = ((uintptr_t)x & (4 * sizeof(T) - 1)) == 0 && ((uintptr_t)y & 15u) == 0;
  if (whole)
    dequantize_kernel<<<pass_grid(n, 256 * 4 * kDequantUnroll), 256, 0, st>>>(x, n, scale, zp, y);
  else
    dequantize_single_kernel<<<grid_for(n, 256 * 4), 256, 0, st>>>(x, n, scale, zp, y);
}

int launch_quantize_with_params(const float *x, int64_t n, uint8_t *y,
    const float *params, cudaStream_t st) {
  const int unroll = quant_unroll(n);
  const int grid = pass_grid(n, kDqlThreads * 4 * unroll);
  OMCUDA_CHECK(launch_pdl(quantize_kernel<false>, grid, kDqlThreads, 0, st, 0,
      pdl_pays(n), x, n, y, params, nullptr, nullptr, 1, nullptr, QuantOutputs{},
      quant_mode(), unroll));
  OMCUDA_CHECK_LAUNCH("quantize_kernel");
  return OMCUDA_OK;
}

int launch_quantize_rows(const float *x, int64_t rows, int64_t cols, int64_t pitch,
    uint8_t *y, int32_t *rowsum, const float *params, cudaStream_t st) {
  const int64_t cap = (int64_t)sm_count() * 8;
  OMCUDA_CHECK(launch_pdl(quantize_rows_kernel, (unsigned)(rows < cap ? rows : cap),
      kDqlThreads, 0, st, 0, pdl_pays(rows * cols), x, rows, (int)cols, (int)pitch, y,
      rowsum, params, quant_mode()));
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
    if (cudaFuncSetAttribute(dql_small_kernel<2>,
            cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaFuncSetAttribute(dql_small_kernel<kSmallMaxWords>,
            cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&a, dql_small_kernel<2>, &q) == cudaSuccess &&
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
  // Four words per thread: 262144 values take 10.3 us this way and 13.3 in three
  // launches.  With sixteen (524288 values, 512 threads) the few SMs of one
  // cluster were slower than the whole machine in three, 18.1 against 14.7 us.
  return rows <= (1 << 20) && pitch <= (1 << 20) &&
         rows * ceil_div(pitch, 4) <=
             (int64_t)small_cluster_limit() * kSmallThreads * kSmallMaxWords;
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
  // Two words per thread while the cluster can still grow.
  int ctas = 1;
  while (ctas < small_cluster_limit() && ctas * kSmallThreads * 2 < p.words)
    ctas *= 2;
  OMCUDA_CHECK(launch_pdl(p.words <= ctas * kSmallThreads * 2
                              ? dql_small_kernel<2>
                              : dql_small_kernel<kSmallMaxWords>,
      (unsigned)ctas, kSmallThreads, 0, st, (unsigned)ctas, true, p));
  count_launch();
  return OMCUDA_OK;
}

int launch_dql_range(const float *x, int64_t n, void *scratch, float *y_scale,
    uint8_t *y_zp, const float **params, cudaStream_t st) {
  DqlScratch *scr = (DqlScratch *)scratch;
  OMCUDA_CHECK(launch_pdl(dql_minmax_kernel, grid_for(n, kDqlThreads * 16), kDqlThreads,
      0, st, 0, pdl_pays(n), x, n, scr, y_scale, y_zp, quant_mode()));
  OMCUDA_CHECK_LAUNCH("dql_minmax_kernel");
  *params = scr->params;
  return OMCUDA_OK;
}

} // namespace omcuda

using namespace omcuda;

extern "C" int64_t omcudaDevDqlScratchBytes(int64_t) {
  return (int64_t)sizeof(DqlScratch);
}

extern "C" int omcudaDevDynamicQuantizeLinear(const float *x, int64_t n,
    uint8_t *y, float *y_scale, uint8_t *y_zp, void *scratch, void *stream) {
  if (n < 0 || (n > 0 && (!x || !y)) || !scratch)
    return fail(OMCUDA_EINVAL, "DynamicQuantizeLinear: bad argument");
  cudaStream_t st = (cudaStream_t)stream;
  if (dql_small_wanted(1, n))
    return launch_dql_small(x, 1, n, n, y, nullptr, y_scale, y_zp, st);
  const float *params = nullptr;
  int rc = launch_dql_range(x, n, scratch, y_scale, y_zp, &params, st);
  if (rc != OMCUDA_OK)
    return rc;
  if (n > 0)
    return launch_quantize_with_params(x, n, y, params, st);
  return OMCUDA_OK;
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
  const int unroll = quant_unroll(n);
  const int grid = pass_grid(n, kDqlThreads * 4 * unroll);
  QuantOutputs outs{params, y_scale, y_zp};
  OMCUDA_CHECK(launch_pdl(quantize_kernel<false>, grid, kDqlThreads, 0, st, 0,
      pdl_pays(n), x, n, y, nullptr, nullptr, nullptr, 1, (const uint32_t *)range, outs,
      quant_mode(), unroll));
  OMCUDA_CHECK_LAUNCH("quantize_kernel");
  return OMCUDA_OK;
}

extern "C" int omcudaDevQuantizeLinear(const float *x, int64_t n, void *y,
    int y_signed, const float *scale, const void *zp, void *stream) {
  if (n < 0 || (n > 0 && (!x || !y)) || !scale)
    return fail(OMCUDA_EINVAL, "QuantizeLinear: bad argument");
  if (n == 0)
    return OMCUDA_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int unroll = quant_unroll(n);
  const int grid = pass_grid(n, kDqlThreads * 4 * unroll);
  if (y_signed)
    OMCUDA_CHECK(launch_pdl(quantize_kernel<true>, grid, kDqlThreads, 0, st, 0,
        pdl_pays(n), x, n, (uint8_t *)y, nullptr, scale, zp, zp != nullptr, nullptr,
        QuantOutputs{}, quant_mode(), unroll));
  else
    OMCUDA_CHECK(launch_pdl(quantize_kernel<false>, grid, kDqlThreads, 0, st, 0,
        pdl_pays(n), x, n, (uint8_t *)y, nullptr, scale, zp, zp != nullptr, nullptr,
        QuantOutputs{}, quant_mode(), unroll));
  OMCUDA_CHECK_LAUNCH("quantize_kernel");
  return OMCUDA_OK;
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
