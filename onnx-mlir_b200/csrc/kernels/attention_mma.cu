// Tensor-core attention for the encoder graphs: softmax(Q K^T * scale) V per
// (batch, head), fp32 in and out, with the matrix products on the warp-level
// tensor-core path (mma.sync m16n8k16, bf16 operands, fp32 accumulators).
//
// It replaces, for head sizes that are multiples of 16 up to 128, the chain the
// reference lowers with CPU loops: two batched fp32 MatMuls
// (src/Conversion/ONNXToKrnl/Math/MatMul.cpp:488-507), a Mul by a constant and
// a Softmax over the last axis (src/Conversion/ONNXToKrnl/Math/Softmax.cpp:25-134).
//
// Accuracy: every fp32 operand a is split as a = hi + lo with hi = bf16(a),
// lo = bf16(a - hi), and each product block is computed as
// hi*hi + lo*hi + hi*lo, which leaves a relative error of about 2^-16 per
// product -- far inside the 1e-3 parity tolerance of the fp32 ops -- while the
// accumulation stays in fp32.  The softmax is computed online over key blocks
// (running maximum and sum, rescaling the accumulator), which is the same
// function as the reference's three-loop form up to fp32 rounding.
//
// Layout: Q, K, V, out are [B, S, *] row-major with row pitches ld_in / ld_out
// (so a fused [T, 3H] QKV buffer is read in place); head h owns columns
// [h*DH, (h+1)*DH).  One CTA = 64 query rows of one (b, h) (4 warps x 16 rows);
// K and V stream through shared memory in blocks of 64 keys as bf16 hi/lo
// pairs.  Scores never leave registers.
#include <cuda_bf16.h>

#include <cstdlib>
#include <cstring>

#include "../common.cuh"
#include "../runtime/internal.h"

namespace omcuda {

namespace {

constexpr int kQRows = 64;  // query rows per CTA
constexpr int kKeys = 64;   // keys per block
constexpr int kPad = 8;     // bf16 elements of row padding (bank spread)

__device__ __forceinline__ void split_bf16(float a, __nv_bfloat16 &hi,
    __nv_bfloat16 &lo) {
  hi = __float2bfloat16_rn(a);
  lo = __float2bfloat16_rn(__fsub_rn(a, __bfloat162float(hi)));
}

__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 a, __nv_bfloat16 b) {
  return (uint32_t)__bfloat16_as_ushort(a) |
         ((uint32_t)__bfloat16_as_ushort(b) << 16);
}

// Splits two floats into packed {hi0,hi1} and {lo0,lo1}.
__device__ __forceinline__ void split2(float x, float y, uint32_t &hi,
    uint32_t &lo) {
  __nv_bfloat16 xh, xl, yh, yl;
  split_bf16(x, xh, xl);
  split_bf16(y, yh, yl);
  hi = pack_bf16(xh, yh);
  lo = pack_bf16(xl, yl);
}

// The same with packed conversions (the kernel for fp32 operands is faster without).
__device__ __forceinline__ void split2_packed(float x, float y, uint32_t &hi,
    uint32_t &lo) {
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(y), "f"(x));
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;"
      : "=r"(lo)
      : "f"(__fsub_rn(y, __uint_as_float(hi & 0xffff0000u))),
        "f"(__fsub_rn(x, __uint_as_float(hi << 16))));
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4],
    uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t &r0,
    uint32_t &r1, uint32_t &r2, uint32_t &r3) {
  asm volatile(
      "ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
      : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
      : "r"(addr));
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t &r0,
    uint32_t &r1, uint32_t &r2, uint32_t &r3) {
  asm volatile(
      "ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
      : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
      : "r"(addr));
}

// 16 bytes from global to shared memory, or zeros.
__device__ __forceinline__ void copy16_async(uint32_t dst, const void *src, bool exists) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
               "r"(exists ? 16 : 0)
               : "memory");
}

// Where the operands lie: fp32, row pitch ld.
struct AttOperands {
  const float *q, *k, *v;
  int64_t ld;
};

template <int DH>
__global__ void __launch_bounds__(128)
    attention_mma_kernel(AttOperands in, int64_t S, int64_t heads, float scale,
        float *__restrict__ out, int64_t ld_out, uint32_t *__restrict__ out_range) {
  constexpr int LD = DH + kPad;  // smem row pitch in bf16 elements
  constexpr int KS = DH / 16;    // k-steps over the head dimension
  constexpr int NT_O = DH / 8;   // n-tiles of the output
  constexpr int NT_S = kKeys / 8;

  extern __shared__ __align__(16) __nv_bfloat16 att_smem[];
  __shared__ RangeBlock range;
  if (threadIdx.x == 0)
    range_block_init(range, blockDim.x >> 5); // (barriers follow)
  pdl_sync();
  in.q = after_pdl(in.q);
  in.k = after_pdl(in.k);
  in.v = after_pdl(in.v);

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int64_t bh = blockIdx.y;
  const int64_t b = bh / heads, h = bh % heads;
  const int64_t q0 = (int64_t)blockIdx.x * kQRows + warp * 16;
  const int64_t ld_in = in.ld;
  const float *Qb = in.q + (b * S) * ld_in + h * DH;
  const float *Kb = in.k + (b * S) * ld_in + h * DH;
  const float *Vb = in.v + (b * S) * ld_in + h * DH;

  // Q fragments (A operand), split once: rows q0+g and q0+g+8.
  uint32_t qh[KS][4], ql[KS][4];
  {
    const int64_t r0 = q0 + g, r1 = q0 + g + 8;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      const int c = ks * 16 + 2 * t;
      float2 v00 = make_float2(0.f, 0.f), v10 = v00, v01 = v00, v11 = v00;
      if (r0 < S) {
        v00 = *reinterpret_cast<const float2 *>(Qb + r0 * ld_in + c);
        v01 = *reinterpret_cast<const float2 *>(Qb + r0 * ld_in + c + 8);
      }
      if (r1 < S) {
        v10 = *reinterpret_cast<const float2 *>(Qb + r1 * ld_in + c);
        v11 = *reinterpret_cast<const float2 *>(Qb + r1 * ld_in + c + 8);
      }
      split2(v00.x, v00.y, qh[ks][0], ql[ks][0]);
      split2(v10.x, v10.y, qh[ks][1], ql[ks][1]);
      split2(v01.x, v01.y, qh[ks][2], ql[ks][2]);
      split2(v11.x, v11.y, qh[ks][3], ql[ks][3]);
    }
  }

  float o[NT_O][4];
#pragma unroll
  for (int i = 0; i < NT_O; ++i)
    o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
  float m0 = -INFINITY, m1 = -INFINITY; // running max of rows g and g+8
  float l0 = 0.0f, l1 = 0.0f;           // running sums

  for (int64_t j0 = 0; j0 < S; j0 += kKeys) {
    // [hi|lo][key][dh] for K, then the same for V
    __nv_bfloat16 (*sK)[kKeys * LD] = reinterpret_cast<__nv_bfloat16 (*)[kKeys * LD]>(att_smem);
    __nv_bfloat16 (*sV)[kKeys * LD] = sK + 2;
    __syncthreads(); // previous block's fragments are no longer read
    {
      // Stage K and V rows j0..j0+63 as bf16 hi/lo, the loads of four trips
      // together.  64 x 500 tokens, 12 heads of 64: 1009 us with ldmatrix
      // below and one trip at a time, 831 with plain loads below, 688 with
      // both; 8 x 512, 8 heads of 128: 131, 132, 121.
#pragma unroll 4
      for (int i = threadIdx.x; i < kKeys * (DH / 4); i += 128) {
        const int key = i / (DH / 4), c4 = (i % (DH / 4)) * 4;
        float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), vv = kv;
        if (j0 + key < S) {
          kv = *reinterpret_cast<const float4 *>(Kb + (j0 + key) * ld_in + c4);
          vv = *reinterpret_cast<const float4 *>(Vb + (j0 + key) * ld_in + c4);
        }
        uint32_t h0, l0w, h1, l1w;
        split2(kv.x, kv.y, h0, l0w);
        split2(kv.z, kv.w, h1, l1w);
        *reinterpret_cast<uint2 *>(&sK[0][key * LD + c4]) = make_uint2(h0, h1);
        *reinterpret_cast<uint2 *>(&sK[1][key * LD + c4]) = make_uint2(l0w, l1w);
        split2(vv.x, vv.y, h0, l0w);
        split2(vv.z, vv.w, h1, l1w);
        *reinterpret_cast<uint2 *>(&sV[0][key * LD + c4]) = make_uint2(h0, h1);
        *reinterpret_cast<uint2 *>(&sV[1][key * LD + c4]) = make_uint2(l0w, l1w);
      }
    }
    __syncthreads();

    // S = Q K^T for this warp's 16 rows x 64 keys.
    float s[NT_S][4];
#pragma unroll
    for (int nt = 0; nt < NT_S; ++nt)
      s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
#pragma unroll
      for (int nt = 0; nt < NT_S; ++nt) {
        uint32_t bh0, bh1, bl0, bl1;
        {
          // Plain loads here: these the compiler may move ahead among the MMAs,
          // which the fp32 form needs, with the conversions between its barriers.
          const int off = (nt * 8 + g) * LD + ks * 16 + 2 * t;
          bh0 = *reinterpret_cast<const uint32_t *>(&sK[0][off]);
          bh1 = *reinterpret_cast<const uint32_t *>(&sK[0][off + 8]);
          bl0 = *reinterpret_cast<const uint32_t *>(&sK[1][off]);
          bl1 = *reinterpret_cast<const uint32_t *>(&sK[1][off + 8]);
        }
        mma_bf16(s[nt], ql[ks], bh0, bh1); // small terms first
        mma_bf16(s[nt], qh[ks], bl0, bl1);
        mma_bf16(s[nt], qh[ks], bh0, bh1);
      }
    }
    // Scale (the graph's Mul by a constant), mask keys past S, block maxima.
    float bm0 = -INFINITY, bm1 = -INFINITY;
#pragma unroll
    for (int nt = 0; nt < NT_S; ++nt) {
      const int64_t key = j0 + nt * 8 + 2 * t;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float v = __fmul_rn(s[nt][e], scale);
        if (key + (e & 1) >= S)
          v = -INFINITY;
        s[nt][e] = v;
      }
      bm0 = fmaxf(bm0, fmaxf(s[nt][0], s[nt][1]));
      bm1 = fmaxf(bm1, fmaxf(s[nt][2], s[nt][3]));
    }
    bm0 = fmaxf(bm0, __shfl_xor_sync(0xffffffffu, bm0, 1));
    bm0 = fmaxf(bm0, __shfl_xor_sync(0xffffffffu, bm0, 2));
    bm1 = fmaxf(bm1, __shfl_xor_sync(0xffffffffu, bm1, 1));
    bm1 = fmaxf(bm1, __shfl_xor_sync(0xffffffffu, bm1, 2));
    const float mn0 = fmaxf(m0, bm0), mn1 = fmaxf(m1, bm1);
    // exp(-inf - finite) = 0 covers the first block; every block holds at
    // least one unmasked key, so mn0 / mn1 are finite.
    const float r0 = expf(m0 - mn0), r1 = expf(m1 - mn1);
    m0 = mn0;
    m1 = mn1;
    float ps0 = 0.0f, ps1 = 0.0f;
#pragma unroll
    for (int nt = 0; nt < NT_S; ++nt) {
      s[nt][0] = expf(s[nt][0] - mn0);
      s[nt][1] = expf(s[nt][1] - mn0);
      s[nt][2] = expf(s[nt][2] - mn1);
      s[nt][3] = expf(s[nt][3] - mn1);
      ps0 += s[nt][0] + s[nt][1];
      ps1 += s[nt][2] + s[nt][3];
    }
    ps0 += __shfl_xor_sync(0xffffffffu, ps0, 1);
    ps0 += __shfl_xor_sync(0xffffffffu, ps0, 2);
    ps1 += __shfl_xor_sync(0xffffffffu, ps1, 1);
    ps1 += __shfl_xor_sync(0xffffffffu, ps1, 2);
    l0 = l0 * r0 + ps0;
    l1 = l1 * r1 + ps1;
#pragma unroll
    for (int i = 0; i < NT_O; ++i) {
      o[i][0] *= r0;
      o[i][1] *= r0;
      o[i][2] *= r1;
      o[i][3] *= r1;
    }
    // O += P V.  The accumulator layout of two adjacent score tiles is the A
    // operand layout of one 16-key step.
#pragma unroll
    for (int kk = 0; kk < kKeys / 16; ++kk) {
      uint32_t ph[4], pl[4];
      split2(s[2 * kk][0], s[2 * kk][1], ph[0], pl[0]);
      split2(s[2 * kk][2], s[2 * kk][3], ph[1], pl[1]);
      split2(s[2 * kk + 1][0], s[2 * kk + 1][1], ph[2], pl[2]);
      split2(s[2 * kk + 1][2], s[2 * kk + 1][3], ph[3], pl[3]);
      // ldmatrix.trans: lane supplies the row (key) address of one 8x8 block:
      // blocks 0,1 = keys kk*16 + {0..7, 8..15} at dh tile d, blocks 2,3 the
      // same keys at dh tile d+1.
      const int mrow = kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
      const int mcol = (lane >> 4) * 8;
#pragma unroll
      for (int d = 0; d < NT_O; d += 2) {
        uint32_t vh0, vh1, vh2, vh3, vl0, vl1, vl2, vl3;
        const int off = mrow * LD + d * 8 + mcol;
        ldmatrix_x4_trans((uint32_t)__cvta_generic_to_shared(&sV[0][off]), vh0,
            vh1, vh2, vh3);
        ldmatrix_x4_trans((uint32_t)__cvta_generic_to_shared(&sV[1][off]), vl0,
            vl1, vl2, vl3);
        mma_bf16(o[d], pl, vh0, vh1);
        mma_bf16(o[d], ph, vl0, vl1);
        mma_bf16(o[d], ph, vh0, vh1);
        mma_bf16(o[d + 1], pl, vh2, vh3);
        mma_bf16(o[d + 1], ph, vl2, vl3);
        mma_bf16(o[d + 1], ph, vh2, vh3);
      }
    }
  }

  // Normalise and store; fold the outputs into the running range.
  float lo = INFINITY, hi = -INFINITY;
  const float inv0 = __fdiv_rn(1.0f, l0), inv1 = __fdiv_rn(1.0f, l1);
  const int64_t r0 = q0 + g, r1 = q0 + g + 8;
  float *ob = out + (b * S) * ld_out + h * DH;
#pragma unroll
  for (int i = 0; i < NT_O; ++i) {
    const int c = i * 8 + 2 * t;
    if (r0 < S) {
      float2 v = make_float2(o[i][0] * inv0, o[i][1] * inv0);
      *reinterpret_cast<float2 *>(ob + r0 * ld_out + c) = v;
      lo = fminf(lo, fminf(v.x, v.y));
      hi = fmaxf(hi, fmaxf(v.x, v.y));
    }
    if (r1 < S) {
      float2 v = make_float2(o[i][2] * inv1, o[i][3] * inv1);
      *reinterpret_cast<float2 *>(ob + r1 * ld_out + c) = v;
      lo = fminf(lo, fminf(v.x, v.y));
      hi = fmaxf(hi, fmaxf(v.x, v.y));
    }
  }
  if (out_range)
    range_commit_block(range, out_range, lo, hi, blockIdx.y * gridDim.x + blockIdx.x);
}

// The bf16 hi / lo planes of a fused projection, with the columns of Q, K and V in a row.
struct AttPlanes {
  const __nv_bfloat16 *hi, *lo;
  int64_t q_col, k_col, v_col;
  int64_t ld;
};

// The same for operands that arrive already split (the projection's GEMM writes the
// same hi and lo that the kernel above would make): a block of keys is 2048 16-byte
// asynchronous copies, and the next block's are in flight during this block's math,
// where above every one of the S / 64 CTAs of a head converts all of its K and V.  Same
// products in the same order: the same bits.  Encoder base, 100 x 500 tokens: 27.0 -> 22.2
// ms; 8 x 400 2.69 -> 2.36 ms.
// Products of four tiles of scores (or output columns) are interleaved, so that one does
// not wait for the one before it: encoder base 20 x 500 tokens 4610 -> 4450 us, large 8 x
// 300 3680 -> 3600.
// kShared: two warps to 16 query rows instead of one.  What a block of keys takes is one
// warp's chain of some 1500 instructions, and one CTA of four warps leaves a scheduler
// nothing else to do: each of the two takes half of the keys for the scores and their
// exponentials, then half of the output columns, and they exchange maxima, sums and P
// through shared memory.  Every value is made by the same operations in the same
// order.  kTiles: tiles of 16 query rows per CTA.
template <bool kShared, int kTiles>
__global__ void __launch_bounds__(32 * kTiles * (kShared ? 2 : 1))
    attention_planes_kernel(AttPlanes in, int64_t S, int64_t heads, float scale,
        float *__restrict__ out, int64_t ld_out, uint32_t *__restrict__ out_range) {
  constexpr int DH = 64;
  constexpr int LD = DH + kPad;  // smem row pitch in bf16 elements
  constexpr int KS = DH / 16;    // k-steps over the head dimension
  constexpr int kWarpsPerTile = kShared ? 2 : 1;
  constexpr int NT_O = DH / 8 / kWarpsPerTile;   // n-tiles of the output, this warp's
  constexpr int NT_S = kKeys / 8 / kWarpsPerTile; // of the scores
  constexpr int kThreads = 32 * kTiles * kWarpsPerTile;
  constexpr int kRows = 16 * kTiles; // query rows per CTA
  constexpr int kTogether = 4; // tiles whose products are interleaved

  extern __shared__ __align__(16) __nv_bfloat16 att_smem[];
  __shared__ RangeBlock range;
  if (threadIdx.x == 0)
    range_block_init(range, blockDim.x >> 5); // (barriers follow)
  pdl_sync();
  in.hi = after_pdl(in.hi);
  in.lo = after_pdl(in.lo);
  // two sets of [hi|lo][key][dh] for K, then the same for V
  constexpr int kSet = 4 * kKeys * LD;

  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % kTiles;
  const int half = kShared ? threadIdx.x / (32 * kTiles) : 0; // of the keys, and of the output columns
  const int nt0 = half * NT_S, d_first = half * NT_O;
  // kShared: block maxima [half][rows]; per lane eight sums and four times four words of P
  float *xch_max = reinterpret_cast<float *>(att_smem + 2 * kSet);
  uint4 *xch = reinterpret_cast<uint4 *>(xch_max + 2 * kRows);
  uint4 *xch_mine = xch + ((warp * 2 + half) * 6) * 32 + lane;
  const uint4 *xch_other = xch + ((warp * 2 + (half ^ 1)) * 6) * 32 + lane;
  const auto pair_barrier = [&] {
    asm volatile("bar.sync %0, 64;" ::"r"(warp + 1) : "memory");
  };
  const int g = lane >> 2, t = lane & 3;
  const int64_t bh = blockIdx.y;
  const int64_t b = bh / heads, h = bh % heads;
  const int64_t q0 = (int64_t)blockIdx.x * kRows + warp * 16;
  const int64_t ld_in = in.ld;
  const int64_t row0 = b * S * ld_in + h * DH;
  const __nv_bfloat16 *src[4] = {in.hi + row0 + in.k_col, in.lo + row0 + in.k_col,
      in.hi + row0 + in.v_col, in.lo + row0 + in.v_col};
  // Requests the K and V rows of keys j0 .. j0+63 (zeros past the sequence).
  auto request = [&](int64_t j0, int set) {
    const uint32_t base =
        (uint32_t)__cvta_generic_to_shared(att_smem + (size_t)set * kSet);
    constexpr int kChunks = DH / 8; // 16-byte pieces of a row
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int i = threadIdx.x; i < kKeys * kChunks; i += kThreads) {
        const int key = i / kChunks, c = i % kChunks;
        const bool exists = j0 + key < S;
        copy16_async(base + (uint32_t)((p * kKeys + key) * LD + 8 * c) * 2u,
            src[p] + (exists ? j0 + key : 0) * ld_in + 8 * c, exists);
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  request(0, 0);

  // Q fragments (A operand), split once: rows q0+g and q0+g+8.
  uint32_t qh[KS][4], ql[KS][4];
  {
    const int64_t r0 = q0 + g, r1 = q0 + g + 8;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      const int c = ks * 16 + 2 * t;
      const int64_t col = row0 + in.q_col + c;
#pragma unroll
      for (int e = 0; e < 4; ++e) { // rows g, g + 8; columns c, c + 8
        const int64_t r = (e & 1) ? r1 : r0;
        const int64_t at = col + r * ld_in + (e >> 1) * 8;
        qh[ks][e] = r < S ? __ldg(reinterpret_cast<const unsigned int *>(in.hi + at)) : 0u;
        ql[ks][e] = r < S ? __ldg(reinterpret_cast<const unsigned int *>(in.lo + at)) : 0u;
      }
    }
  }

  float o[NT_O][4];
#pragma unroll
  for (int i = 0; i < NT_O; ++i)
    o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
  float m0 = -INFINITY, m1 = -INFINITY; // running max of rows g and g+8
  float l0 = 0.0f, l1 = 0.0f;           // running sums

  for (int64_t j0 = 0; j0 < S; j0 += kKeys) {
    const int set = (int)((j0 / kKeys) & 1);
    __nv_bfloat16 (*sK)[kKeys * LD] =
        reinterpret_cast<__nv_bfloat16 (*)[kKeys * LD]>(att_smem + (size_t)set * kSet);
    __nv_bfloat16 (*sV)[kKeys * LD] = sK + 2;
    __syncthreads(); // previous block's fragments are no longer read
    if (j0 + kKeys < S) {
      request(j0 + kKeys, set ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();

    // S = Q K^T for this warp's 16 rows x 64 keys.
    float s[NT_S][4];
#pragma unroll
    for (int nt = 0; nt < NT_S; ++nt)
      s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
#pragma unroll
      for (int n0 = 0; n0 < NT_S; n0 += kTogether) {
        uint32_t kf[kTogether][4]; // hi of k 0..7 and 8..15, then lo
#pragma unroll
        for (int i = 0; i < kTogether; ++i) {
          const int nt = nt0 + n0 + i;
          // a lane supplies one key row of one of the four 8x8 blocks
          ldmatrix_x4((uint32_t)__cvta_generic_to_shared(
                          &sK[lane >> 4][(nt * 8 + (lane & 7)) * LD + ks * 16 +
                                         ((lane >> 3) & 1) * 8]),
              kf[i][0], kf[i][1], kf[i][2], kf[i][3]);
        }
        // small terms first; a term of every tile before the next one of any
#pragma unroll
        for (int i = 0; i < kTogether; ++i)
          mma_bf16(s[n0 + i], ql[ks], kf[i][0], kf[i][1]);
#pragma unroll
        for (int i = 0; i < kTogether; ++i)
          mma_bf16(s[n0 + i], qh[ks], kf[i][2], kf[i][3]);
#pragma unroll
        for (int i = 0; i < kTogether; ++i)
          mma_bf16(s[n0 + i], qh[ks], kf[i][0], kf[i][1]);
      }
    }
    // Scale (the graph's Mul by a constant), mask keys past S, block maxima.
    float bm0 = -INFINITY, bm1 = -INFINITY;
    const int left = (int)(S - j0 < kKeys ? S - j0 : kKeys) - 2 * t;
#pragma unroll
    for (int nt = 0; nt < NT_S; ++nt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float v = __fmul_rn(s[nt][e], scale);
        s[nt][e] = (nt0 + nt) * 8 + (e & 1) >= left ? -INFINITY : v;
      }
      bm0 = fmaxf(bm0, fmaxf(s[nt][0], s[nt][1]));
      bm1 = fmaxf(bm1, fmaxf(s[nt][2], s[nt][3]));
    }
    bm0 = fmaxf(bm0, __shfl_xor_sync(0xffffffffu, bm0, 1));
    bm0 = fmaxf(bm0, __shfl_xor_sync(0xffffffffu, bm0, 2));
    bm1 = fmaxf(bm1, __shfl_xor_sync(0xffffffffu, bm1, 1));
    bm1 = fmaxf(bm1, __shfl_xor_sync(0xffffffffu, bm1, 2));
    if (kShared) {
      if (t == 0) {
        xch_max[half * kRows + warp * 16 + g] = bm0;
        xch_max[half * kRows + warp * 16 + g + 8] = bm1;
      }
      pair_barrier();
      bm0 = fmaxf(bm0, xch_max[(half ^ 1) * kRows + warp * 16 + g]);
      bm1 = fmaxf(bm1, xch_max[(half ^ 1) * kRows + warp * 16 + g + 8]);
    }
    const float mn0 = fmaxf(m0, bm0), mn1 = fmaxf(m1, bm1);
    // exp(-inf - finite) = 0 covers the first block; every block holds at
    // least one unmasked key, so mn0 / mn1 are finite.
    const float r0 = expf(m0 - mn0), r1 = expf(m1 - mn1);
    m0 = mn0;
    m1 = mn1;
    float ps0 = 0.0f, ps1 = 0.0f;
    float pair0[NT_S], pair1[NT_S]; // sums of a tile's two values of a row
#pragma unroll
    for (int nt = 0; nt < NT_S; ++nt) {
      s[nt][0] = expf(s[nt][0] - mn0);
      s[nt][1] = expf(s[nt][1] - mn0);
      s[nt][2] = expf(s[nt][2] - mn1);
      s[nt][3] = expf(s[nt][3] - mn1);
      pair0[nt] = s[nt][0] + s[nt][1];
      pair1[nt] = s[nt][2] + s[nt][3];
    }
    // P of 16 keys at a time: the accumulator layout of two adjacent score tiles is the A
    // operand layout of one such step.
    uint32_t ph[kKeys / 16][4], pl[kKeys / 16][4];
    constexpr int kOwn = NT_S / 2; // steps of this warp's keys
#pragma unroll
    for (int k = 0; k < kOwn; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        split2_packed(s[2 * k + (e >> 1)][2 * (e & 1)], s[2 * k + (e >> 1)][2 * (e & 1) + 1], ph[k][e],
            pl[k][e]);
    if constexpr (kShared) {
      static_assert(NT_S == 4 && kOwn == 2, "what a lane hands over");
      const auto bits = [](float a, float b, float c, float d) {
        return make_uint4(__float_as_uint(a), __float_as_uint(b), __float_as_uint(c),
            __float_as_uint(d));
      };
      xch_mine[0] = bits(pair0[0], pair0[1], pair0[2], pair0[3]);
      xch_mine[32] = bits(pair1[0], pair1[1], pair1[2], pair1[3]);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        xch_mine[32 * (2 + 2 * k)] = make_uint4(ph[k][0], ph[k][1], ph[k][2], ph[k][3]);
        xch_mine[32 * (3 + 2 * k)] = make_uint4(pl[k][0], pl[k][1], pl[k][2], pl[k][3]);
      }
      pair_barrier();
      const uint4 a = xch_other[0], c = xch_other[32];
      const float z0[4] = {__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z),
          __uint_as_float(a.w)};
      const float z1[4] = {__uint_as_float(c.x), __uint_as_float(c.y), __uint_as_float(c.z),
          __uint_as_float(c.w)};
#pragma unroll
      for (int i = 0; i < 8; ++i) { // keys in order, whoever made their sums
        const bool mine = (i >> 2) == half;
        ps0 += mine ? pair0[i & 3] : z0[i & 3];
        ps1 += mine ? pair1[i & 3] : z1[i & 3];
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint4 h = xch_other[32 * (2 + 2 * k)], l = xch_other[32 * (3 + 2 * k)];
        const uint32_t hw[4] = {h.x, h.y, h.z, h.w}, lw[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          // step k is half 0's, step 2 + k half 1's
          ph[2 + k][e] = half ? ph[k][e] : hw[e];
          pl[2 + k][e] = half ? pl[k][e] : lw[e];
          ph[k][e] = half ? hw[e] : ph[k][e];
          pl[k][e] = half ? lw[e] : pl[k][e];
        }
      }
    } else {
#pragma unroll
      for (int nt = 0; nt < NT_S; ++nt) {
        ps0 += pair0[nt];
        ps1 += pair1[nt];
      }
    }
    ps0 += __shfl_xor_sync(0xffffffffu, ps0, 1);
    ps0 += __shfl_xor_sync(0xffffffffu, ps0, 2);
    ps1 += __shfl_xor_sync(0xffffffffu, ps1, 1);
    ps1 += __shfl_xor_sync(0xffffffffu, ps1, 2);
    l0 = l0 * r0 + ps0;
    l1 = l1 * r1 + ps1;
#pragma unroll
    for (int i = 0; i < NT_O; ++i) {
      o[i][0] *= r0;
      o[i][1] *= r0;
      o[i][2] *= r1;
      o[i][3] *= r1;
    }
    // O += P V.
#pragma unroll
    for (int kk = 0; kk < kKeys / 16; ++kk) {
      // ldmatrix.trans: lane supplies the row (key) address of one 8x8 block:
      // blocks 0,1 = keys kk*16 + {0..7, 8..15} at dh tile d, blocks 2,3 the
      // same keys at dh tile d+1.
      const int mrow = kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
      const int mcol = (lane >> 4) * 8;
#pragma unroll
      for (int d0 = 0; d0 < NT_O; d0 += kTogether) {
        uint32_t vh[kTogether][2], vl[kTogether][2];
#pragma unroll
        for (int i = 0; i < kTogether; i += 2) {
          const int off = mrow * LD + (d_first + d0 + i) * 8 + mcol;
          ldmatrix_x4_trans((uint32_t)__cvta_generic_to_shared(&sV[0][off]), vh[i][0],
              vh[i][1], vh[i + 1][0], vh[i + 1][1]);
          ldmatrix_x4_trans((uint32_t)__cvta_generic_to_shared(&sV[1][off]), vl[i][0],
              vl[i][1], vl[i + 1][0], vl[i + 1][1]);
        }
#pragma unroll
        for (int i = 0; i < kTogether; ++i)
          mma_bf16(o[d0 + i], pl[kk], vh[i][0], vh[i][1]);
#pragma unroll
        for (int i = 0; i < kTogether; ++i)
          mma_bf16(o[d0 + i], ph[kk], vl[i][0], vl[i][1]);
#pragma unroll
        for (int i = 0; i < kTogether; ++i)
          mma_bf16(o[d0 + i], ph[kk], vh[i][0], vh[i][1]);
      }
    }
  }

  // Normalise and store; fold the outputs into the running range.
  float lo = INFINITY, hi = -INFINITY;
  const float inv0 = __fdiv_rn(1.0f, l0), inv1 = __fdiv_rn(1.0f, l1);
  const int64_t r0 = q0 + g, r1 = q0 + g + 8;
  float *ob = out + (b * S) * ld_out + h * DH;
#pragma unroll
  for (int i = 0; i < NT_O; ++i) {
    const int c = (d_first + i) * 8 + 2 * t;
    if (r0 < S) {
      float2 v = make_float2(o[i][0] * inv0, o[i][1] * inv0);
      *reinterpret_cast<float2 *>(ob + r0 * ld_out + c) = v;
      lo = fminf(lo, fminf(v.x, v.y));
      hi = fmaxf(hi, fmaxf(v.x, v.y));
    }
    if (r1 < S) {
      float2 v = make_float2(o[i][2] * inv1, o[i][3] * inv1);
      *reinterpret_cast<float2 *>(ob + r1 * ld_out + c) = v;
      lo = fminf(lo, fminf(v.x, v.y));
      hi = fmaxf(hi, fmaxf(v.x, v.y));
    }
  }
  if (out_range)
    range_commit_block(range, out_range, lo, hi, blockIdx.y * gridDim.x + blockIdx.x);
}

} // namespace

// True when the tensor-core kernel can take the problem: head size 32, 64 or
// 128 and 8-byte aligned rows.
bool attention_mma_supported(const float *Q, const float *K, const float *V,
    const float *out, int64_t dh, int64_t ld_in, int64_t ld_out) {
  return (dh == 32 || dh == 64 || dh == 128) && (ld_in % 4 == 0) &&
         (ld_out % 2 == 0) &&
         ((((uintptr_t)Q | (uintptr_t)K | (uintptr_t)V) & 15u) == 0) &&
         (((uintptr_t)out & 7u) == 0);
}

// Shared memory beyond 48 KiB has to be asked for once per device and kernel.
template <typename In>
static int launch_mma(void (*kernel)(In, int64_t, int64_t, float, float *, int64_t, uint32_t *),
    PerDeviceInt *attr_set, int rows, unsigned threads, int smem, const In &in, int64_t B, int64_t S,
    int64_t heads, int64_t dh, float scale, float *out, int64_t ld_out, void *out_range,
    cudaStream_t st) {
  const dim3 grid((unsigned)ceil_div(S, rows), (unsigned)(B * heads));
  if (smem > 48 * 1024 && !attr_set->get()) {
    OMCUDA_CHECK(cudaFuncSetAttribute(
        kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr_set->set(1);
  }
  OMCUDA_CHECK(launch_pdl(kernel, grid, threads, (size_t)smem, st, 0,
      pdl_pays(B * S * heads * dh), in, S, heads, scale, out, ld_out, (uint32_t *)out_range));
  OMCUDA_CHECK_LAUNCH("attention_mma_kernel");
  return OMCUDA_OK;
}

template <int DH>
static int launch_mma_f32(const AttOperands &in, int64_t B, int64_t S, int64_t heads,
    float scale, float *out, int64_t ld_out, void *out_range, cudaStream_t st) {
  static PerDeviceInt attr_set;
  return launch_mma(attention_mma_kernel<DH>, &attr_set, kQRows, 128,
      4 * kKeys * (DH + kPad) * (int)sizeof(__nv_bfloat16), in, B, S, heads, DH, scale, out,
      ld_out, out_range, st);
}

template <bool kShared, int kTiles>
static int launch_mma_planes(const AttPlanes &in, int64_t B, int64_t S, int64_t heads,
    float scale, float *out, int64_t ld_out, void *out_range, cudaStream_t st) {
  static PerDeviceInt attr_set;
  return launch_mma(attention_planes_kernel<kShared, kTiles>, &attr_set, 16 * kTiles,
      32 * kTiles * (kShared ? 2 : 1),
      2 * 4 * kKeys * (64 + kPad) * (int)sizeof(__nv_bfloat16) +
          (kShared ? 2 * 16 * kTiles * (int)sizeof(float) +
                         2 * kTiles * 6 * 32 * (int)sizeof(uint4)
                   : 0),
      in, B, S, heads, 64, scale, out, ld_out, out_range, st);
}

int launch_attention_mma(const float *Q, const float *K, const float *V,
    int64_t B, int64_t S, int64_t heads, int64_t dh, float scale, float *out,
    int64_t ld_in, int64_t ld_out, void *out_range, cudaStream_t st) {
  AttOperands in = {};
  in.q = Q;
  in.k = K;
  in.v = V;
  in.ld = ld_in;
  if (dh == 64)
    return launch_mma_f32<64>(in, B, S, heads, scale, out, ld_out, out_range, st);
  if (dh == 32)
    return launch_mma_f32<32>(in, B, S, heads, scale, out, ld_out, out_range, st);
  return launch_mma_f32<128>(in, B, S, heads, scale, out, ld_out, out_range, st);
}

// The form of the kernel that reads planes: head size 64, 16-byte aligned rows.
bool attention_mma_planes_supported(int64_t B, int64_t S, int64_t heads, int64_t dh,
    int64_t ld_planes, int64_t ld_out, const void *hi, const void *lo, const float *out) {
  // OMCUDA_ATTENTION=simt asks for the fp32 kernel, to cross-check them.
  static const bool disabled = [] {
    const char *s = getenv("OMCUDA_ATTENTION");
    return s && strcmp(s, "simt") == 0;
  }();
  return !disabled && dh == 64 && S > 0 && B * heads <= 65535 && ld_planes % 8 == 0 &&
         ld_out % 2 == 0 && (((uintptr_t)hi | (uintptr_t)lo) & 15u) == 0 &&
         ((uintptr_t)out & 7u) == 0;
}

int launch_attention_mma_planes(const void *hi, const void *lo, int64_t ld_planes,
    int64_t q_col, int64_t k_col, int64_t v_col, int64_t B, int64_t S, int64_t heads,
    float scale, float *out, int64_t ld_out, void *out_range, cudaStream_t st) {
  AttPlanes in = {};
  in.hi = (const __nv_bfloat16 *)hi;
  in.lo = (const __nv_bfloat16 *)lo;
  in.q_col = q_col;
  in.k_col = k_col;
  in.v_col = v_col;
  in.ld = ld_planes;
  // Two warps to a tile while all CTAs of that form are resident (two to an SM; of the
  // other three), 32 rows to a CTA while those are, too: the fewer warps an SM has, the
  // less one waits for another's instructions to be fetched and issued.  Encoder runs,
  // one warp to a tile / two, 64 rows / two, 32 rows: base 1 x 476, 180 CTAs of 32 rows,
  // 1049 / 970 / 830 us, 2 x 304, 240, 945 / 896 / 813, 5 x 68 707 / 683 / 642, large 1 x 300
  // 1816 / 1712 / 1524, base 1 x 61 450 / 453 / 442, but 4 x 304, 480, 1169 / 1117 / 1189 and 5 x
  // 304, 300 CTAs of 64 rows, 1212 / 1260.
  const int64_t resident = 2 * sm_count();
  if (ceil_div(S, 32) * B * heads <= resident)
    return launch_mma_planes<true, 2>(in, B, S, heads, scale, out, ld_out, out_range, st);
  if (ceil_div(S, 64) * B * heads <= resident)
    return launch_mma_planes<true, 4>(in, B, S, heads, scale, out, ld_out, out_range, st);
  return launch_mma_planes<false, 4>(in, B, S, heads, scale, out, ld_out, out_range, st);
}

} // namespace omcuda
