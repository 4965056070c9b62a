// Operand preparation for the int8 GEMMs and the SIMT (dp4a) GEMM.
//
// prepare_b: B arrives [K,N] row-major (the ONNX layout of a MatMulInteger /
// QLinearMatMul weight).  Both GEMM kernels consume it K-major, so it is
// copied once into Bt[N][kp] (kp = K rounded up to 16, zero padded) together
// with its column sums, which carry the A zero point through the epilogue
// (see gemm_epilogue.cuh).
//
// gemm_i8_warp_kernel: one warp per output column n and per group of MT rows;
// the 32 lanes split K in 16-byte chunks (coalesced 512-byte reads of the Bt
// row), accumulate with dp4a, and fold with shuffles.  It is the path for
// small M, where the GEMM is bound by reading the weight once from HBM, and
// for shapes the tensor-core kernel does not take (K not a multiple of 16,
// unaligned bases).  Integer accumulation wraps in 32 bits in any order, so
// its results are bit-identical to the tensor-core kernel's.
#include <cstdlib>

#include "../runtime/internal.h"
#include "gemm_epilogue.cuh"

namespace omcuda {

// ---- B preparation -----------------------------------------------------------

// Bound by the read and the write of B.  A thread takes a 4 x 4 block of a 64(k) x
// 64(n) tile: four words of neighbouring columns (or bytes, where rows of B do not
// start on words), turned in registers into words of neighbouring k, which pass
// through shared memory to leave row by row.  With the column sums below 14336 x 4096
// (59 MB) take 40 us; byte by byte, and sums of a column per thread, 485.
__global__ void __launch_bounds__(256)
    transpose_b_kernel(const uint8_t *__restrict__ B, int64_t K, int64_t N,
        int64_t kp, uint8_t *__restrict__ Bt) {
  __shared__ uint32_t tile[64][17]; // [column][word of k]
  const int64_t k0 = (int64_t)blockIdx.y * 64, n0 = (int64_t)blockIdx.x * 64;
  const bool words = (((uintptr_t)B | (uintptr_t)N) & 3u) == 0;
  {
    const int nb = threadIdx.x & 15, kb = threadIdx.x >> 4;
    const int64_t n = n0 + 4 * nb;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t k = k0 + 4 * kb + i;
      w[i] = 0;
      if (k < K && n < N) {
        const uint8_t *src = B + k * N + n;
        if (words) {
          w[i] = __ldcs(reinterpret_cast<const uint32_t *>(src));
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (n + j < N)
              w[i] |= (uint32_t)__ldg(src + j) << (8 * j);
        }
      }
    }
    // 4 x 4 bytes transposed
    const uint32_t a0 = __byte_perm(w[0], w[1], 0x5140), a1 = __byte_perm(w[0], w[1], 0x7362);
    const uint32_t b0 = __byte_perm(w[2], w[3], 0x5140), b1 = __byte_perm(w[2], w[3], 0x7362);
    tile[4 * nb][kb] = __byte_perm(a0, b0, 0x5410);
    tile[4 * nb + 1][kb] = __byte_perm(a0, b0, 0x7632);
    tile[4 * nb + 2][kb] = __byte_perm(a1, b1, 0x5410);
    tile[4 * nb + 3][kb] = __byte_perm(a1, b1, 0x7632);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = (threadIdx.x >> 4) + 16 * i, c = threadIdx.x & 15;
    const int64_t n = n0 + r, k = k0 + 4 * c;
    if (n >= N || k >= kp)
      continue;
    const uint32_t w = tile[r][c];
    uint8_t *dst = Bt + n * kp + k;
    if (((uintptr_t)Bt & 3u) == 0) {
      *reinterpret_cast<uint32_t *>(dst) = w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        dst[j] = (uint8_t)(w >> (8 * j));
    }
  }
}

// QLinearMatMul's column scales (src/Conversion/ONNXToKrnl/Math/QLinearMatMul.cpp:123-138).
__device__ __forceinline__ float requant_scale(const RequantScale &rq, int64_t i) {
  const float *a = after_pdl(rq.a_scale), *b = after_pdl(rq.b_scale), *y = after_pdl(rq.y_scale);
  return __fdiv_rn(__fmul_rn(*a, b[i]), *y);
}

// One warp per row, a 16-byte chunk per lane and trip; with dst, the row is also
// copied into an aligned row of `pitch` bytes whose tail is zero.  The column
// scales of a QLinearMatMul ride along (rq.len != 0) in blocks behind those of
// the rows: a launch of their own was 2.1 us for a few thousand divides, and made
// by the blocks of the rows, one of them for up to 8 rows, they were a serial chain
// (1 x 256 x 32768: 45 us a call so, 19 now).
//
// The sums serve the zero points of the weight, which are mostly all zero: with zp
// (zp_len bytes), a block first looks at those and leaves its sums as they are if it
// finds nothing else.  The tails still load them, whatever they hold, and multiply
// them by those zeros modulo 2^32.  QLinearMatMul 512 x 1024 x 1024 12.3 -> 8.3 us a
// call, together with the launch that overlaps; 16384 x 1024 x 4096 with changing
// inputs 100.2 -> 82.5, together with the GEMM's tail.
template <bool kSigned>
__global__ void __launch_bounds__(256)
    rowsum_kernel(const uint8_t *__restrict__ A, int64_t M, int64_t K,
        int32_t *__restrict__ rowsum, uint8_t *__restrict__ dst, int64_t pitch,
        const uint8_t *__restrict__ zp, int64_t zp_len, RequantScale rq) {
  pdl_sync();
  A = after_pdl(A);
  zp = after_pdl(zp);
  const int64_t row_blocks = ceil_div(M, (int64_t)(blockDim.x >> 5));
  if (blockIdx.x >= row_blocks) {
    const int64_t i = ((int64_t)blockIdx.x - row_blocks) * blockDim.x + threadIdx.x;
    if (i < rq.len)
      rq.S[i] = requant_scale(rq, i);
    return;
  }
  if (zp) {
    uint32_t any = 0;
    for (int64_t i = 16 * (int64_t)threadIdx.x; i < zp_len; i += 16 * 256) {
      if ((((uintptr_t)zp) & 15u) == 0 && i + 16 <= zp_len) {
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(zp + i));
        any |= q.x | q.y | q.z | q.w;
      } else {
        for (int64_t j = i; j < i + 16 && j < zp_len; ++j)
          any |= __ldg(zp + j);
      }
    }
    if (!__syncthreads_or((int)any)) {
      if (!dst)
        return;
      rowsum = nullptr;
    }
  }
  const int64_t m = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (m >= M)
    return;
  const int lane = threadIdx.x & 31;
  const uint8_t *row = A + m * K;
  const bool vec = (((uintptr_t)row) & 15u) == 0;
  int32_t s = 0;
#pragma unroll 4
  for (int64_t k = 16 * lane; k < K; k += 512) {
    uint32_t w[4];
    if (vec && k + 16 <= K) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(row + k));
      w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
    } else {
      load_bytes(row + k, (int)(K - k < 16 ? K - k : 16), w);
    }
    if (dst)
      *reinterpret_cast<uint4 *>(dst + m * pitch + k) = make_uint4(w[0], w[1], w[2], w[3]);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      s = add_bytes<kSigned>(w[j], s);
  }
  if (!rowsum)
    return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0)
    rowsum[m] = s;
}

__global__ void requant_scale_kernel(RequantScale rq) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < rq.len)
    rq.S[i] = requant_scale(rq, i);
}

// ---- SIMT GEMM ----------------------------------------------------------------

template <bool kASigned, bool kBSigned>
__device__ __forceinline__ int32_t dp4a_mixed(uint32_t a, uint32_t b, int32_t c) {
  int32_t d;
  if (kASigned && kBSigned)
    asm("dp4a.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  else if (kASigned && !kBSigned)
    asm("dp4a.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  else if (!kASigned && kBSigned)
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  else
    asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// 16 bytes of row m of A from K offset k0 on, zeros beyond the matrix.  vec_ok:
// rows are 16-byte aligned and, where K ends inside a chunk, zero up to its end.
__device__ __forceinline__ uint4 load_a_chunk(const uint8_t *__restrict__ A,
    int64_t m, const EpiParams &p, int64_t k0, bool vec_ok) {
  if (m >= p.M || k0 >= p.K)
    return make_uint4(0, 0, 0, 0);
  const uint8_t *src = A + m * p.lda + k0;
  if (vec_ok)
    return __ldg(reinterpret_cast<const uint4 *>(src));
  uint32_t w[4];
  load_bytes(src, (int)(p.K - k0 < 16 ? p.K - k0 : 16), w);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

template <int MT, bool kASigned, bool kBSigned>
__global__ void __launch_bounds__(256)
    gemm_i8_warp_kernel(const uint8_t *__restrict__ A,
        const uint8_t *__restrict__ Bt, int64_t kp, EpiParams p) {
  const int lane = threadIdx.x & 31;
  const int64_t n = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t m0 = (int64_t)blockIdx.y * MT;
  if (n >= p.N)
    return; // whole warp leaves together
  const bool vec_ok = ((p.lda & 15) == 0) && (((uintptr_t)A & 15u) == 0);
  int32_t acc[MT];
#pragma unroll
  for (int i = 0; i < MT; ++i)
    acc[i] = 0;
  const uint4 *brow = reinterpret_cast<const uint4 *>(Bt + n * kp);
  const int64_t chunks = kp >> 4;
  for (int64_t c = lane; c < chunks; c += 32) {
    uint4 b = __ldg(brow + c);
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      uint4 a = load_a_chunk(A, m0 + i, p, c << 4, vec_ok);
      int32_t s = acc[i];
      s = dp4a_mixed<kASigned, kBSigned>(a.x, b.x, s);
      s = dp4a_mixed<kASigned, kBSigned>(a.y, b.y, s);
      s = dp4a_mixed<kASigned, kBSigned>(a.z, b.z, s);
      s = dp4a_mixed<kASigned, kBSigned>(a.w, b.w, s);
      acc[i] = s;
    }
  }
#pragma unroll
  for (int i = 0; i < MT; ++i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
  }
  // Lane i finishes row m0+i (MT <= 32).
  const EpiScalars sc = epi_scalars(p);
  float lo = INFINITY, hi = -INFINITY;
  int32_t mine = 0;
#pragma unroll
  for (int i = 0; i < MT; ++i)
    if (lane == i)
      mine = acc[i];
  const int64_t m = m0 + lane;
  if (lane < MT && m < p.M) {
    EpiRow row = epi_row(p, m);
    int32_t v = epi_int(p, row, mine, n);
    if (p.kind == OMCUDA_EPI_I32) {
      reinterpret_cast<int32_t *>(p.Y)[m * p.N + n] = v;
    } else if (p.kind == OMCUDA_EPI_DEQUANT) {
      float y = epi_dequant(p, sc, v, n);
      if (p.residual)
        y = __fadd_rn(y, __ldg(p.residual + m * p.N + n));
      reinterpret_cast<float *>(p.Y)[m * p.N + n] = y;
      lo = fminf(lo, y);
      hi = fmaxf(hi, y);
    } else {
      reinterpret_cast<uint8_t *>(p.Y)[m * p.N + n] =
          (uint8_t)epi_requant(p, sc, v, n);
    }
  }
  if (p.out_range && p.kind == OMCUDA_EPI_DEQUANT)
    range_commit_warp(p.out_range, lo, hi);
}


// ---- GEMV-shaped GEMM for M <= 16 ----------------------------------------------
//
// With a handful of rows the GEMM is one pass over the K*N bytes of the
// weight: HBM bound.  A block of kWarps warps owns CB adjacent output
// columns (CB rows of Bt) and MT rows of A, and splits K between its warps:
// chunk c (16 bytes of K) goes to thread c mod (32 * kWarps), so that a
// warp-wide load of Bt is one coalesced 512-byte access and every SM keeps
// tens of kilobytes of weight reads in flight (CB loads per thread and trip,
// trips unrolled by two).  A is tiny (M*K bytes) and is served by L1; loading
// one A chunk for CB columns keeps the L1 traffic per weight byte at MT / CB.
// The partial sums are folded with shuffles inside each warp and through
// shared memory between the warps (no global workspace, no atomics); the
// first MT * CB threads of the block run the epilogue.  Integer addition is
// exact in any order, so the result equals the other kernels' bit for bit.
// How many warps: see gemv_warps().
constexpr int kGemvSmWarps = 32; // resident per SM: 64 registers a thread

// Asks for `cols` columns of the weight (rows of Bt, kp bytes each) in L2.  The
// GEMV-shaped kernels do this before pdl_sync(): their blocks are resident while
// the activation is still being quantized, and the weight, which is all they
// have to wait for, is on its way by then.  A prefetch reads nothing, so it does
// not matter whether the weight has been written yet.  Weights of more than
// half of L2 would be evicted before they are read: those are left alone.
// Linear 16 x 14336 x 4096 28.7 -> 24.6 us, 1 x 4096 x 14336 18.4 -> 17.7 when they came.
__device__ __forceinline__ void prefetch_weight(
    const uint8_t *Bt, int64_t kp, int64_t n0, int cols, int64_t N) {
  const int j = threadIdx.x;
  if (j < cols && n0 + j < N && N * kp <= ((int64_t)64 << 20))
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(Bt + (n0 + j) * kp),
                 "r"((uint32_t)kp)
                 : "memory");
}

template <int MT, int CB, int kWarps, bool kASigned, bool kBSigned>
__global__ void __launch_bounds__(32 * kWarps)
    gemm_i8_gemv_kernel(const uint8_t *__restrict__ A,
        const uint8_t *__restrict__ Bt, int64_t kp, EpiParams p) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t m0 = (int64_t)blockIdx.y * MT;
  const bool vec_ok = ((p.lda & 15) == 0) && (((uintptr_t)A & 15u) == 0);
  const int64_t chunks = kp >> 4;
  constexpr int kStep = 32 * kWarps;
  __shared__ int32_t part[kWarps][MT * CB];
  static_assert(MT * CB <= 32, "the epilogue runs in the first warp");
  float lo = INFINITY, hi = -INFINITY;
  // A block walks column groups (grid-stride), so that a launch is a few
  // resident blocks per SM streaming the weight rather than thousands of
  // short-lived ones.
  const int64_t groups = ceil_div(p.N, CB);
  for (int64_t g = blockIdx.x; g < groups; g += gridDim.x)
    prefetch_weight(Bt, kp, g * CB, CB, p.N);
  if (p.early_next)
    pdl_sync();
  else
    pdl_wait();
  // (opaque: with after_pdl the compiler overlaps trips and takes 94 registers
  // instead of 64, and 1 x 4096 x 14336 went from 17.7 to 18.5 us in blocks of four warps)
  A = after_pdl_opaque(A);
  Bt = after_pdl_opaque(Bt);
  const EpiScalars sc = epi_scalars(p);
  for (int64_t g = blockIdx.x; g < groups; g += gridDim.x) {
    const int64_t n0 = g * CB;
    int32_t acc[MT][CB];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < CB; ++j)
        acc[i][j] = 0;
    const uint4 *brow[CB];
#pragma unroll
    for (int j = 0; j < CB; ++j) // columns past N re-read the last one; never stored
      brow[j] = reinterpret_cast<const uint4 *>(Bt + (n0 + j < p.N ? n0 + j : p.N - 1) * kp);
    auto consume = [&](int64_t c, const uint4 (&b)[CB]) {
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const uint4 a = load_a_chunk(A, m0 + i, p, c << 4, vec_ok);
#pragma unroll
        for (int j = 0; j < CB; ++j) {
          int32_t s = acc[i][j];
          s = dp4a_mixed<kASigned, kBSigned>(a.x, b[j].x, s);
          s = dp4a_mixed<kASigned, kBSigned>(a.y, b[j].y, s);
          s = dp4a_mixed<kASigned, kBSigned>(a.z, b[j].z, s);
          s = dp4a_mixed<kASigned, kBSigned>(a.w, b[j].w, s);
          acc[i][j] = s;
        }
      }
    };
    int64_t c = threadIdx.x;
    for (; c + kStep < chunks; c += 2 * kStep) {
      uint4 b0[CB], b1[CB];
#pragma unroll
      for (int j = 0; j < CB; ++j) {
        b0[j] = __ldcs(brow[j] + c);
        b1[j] = __ldcs(brow[j] + c + kStep);
      }
      consume(c, b0);
      consume(c + kStep, b1);
    }
    if (c < chunks) {
      uint4 b0[CB];
#pragma unroll
      for (int j = 0; j < CB; ++j)
        b0[j] = __ldcs(brow[j] + c);
      consume(c, b0);
    }
    // The lanes' sums of all kSums outputs: while a lane holds several, it sends half of
    // them away and adds what it gets to the other half (six shuffles for four sums, one
    // by one twenty).
    constexpr int kSums = MT * CB;
    static_assert((kSums & (kSums - 1)) == 0, "halved until one is left");
    int32_t v[kSums];
#pragma unroll
    for (int i = 0; i < kSums; ++i)
      v[i] = acc[i / CB][i % CB];
#pragma unroll
    for (int step = 0; step < 5; ++step) {
      const int o = 16 >> step, left = kSums >> (step + 1);
      if (left > 0) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < left; ++j) {
          const int32_t sent = upper ? v[j] : v[j + left];
          v[j] = (upper ? v[j + left] : v[j]) + __shfl_xor_sync(0xffffffffu, sent, o);
        }
      } else {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
      }
    }
    if (lane % (32 / kSums) == 0)
      part[warp][lane / (32 / kSums)] = v[0];
    __syncthreads();
    // Thread t of the first warp finishes output (row m0 + t / CB, column n0 + t % CB).
    if (warp == 0) {
      const int64_t m = m0 + lane / CB, n = n0 + lane % CB;
      if (lane < MT * CB && m < p.M && n < p.N) {
        int32_t sum = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w)
          sum += part[w][lane];
        const EpiParams e = epi_after_pdl(p);
        const EpiRow row = epi_row(e, m);
        const int32_t v = epi_int(e, row, sum, n);
        if (p.kind == OMCUDA_EPI_I32) {
          reinterpret_cast<int32_t *>(p.Y)[m * p.N + n] = v;
        } else if (p.kind == OMCUDA_EPI_DEQUANT) {
          float y = epi_dequant(e, sc, v, n);
          if (e.residual)
            y = __fadd_rn(y, __ldg(e.residual + m * p.N + n));
          reinterpret_cast<float *>(p.Y)[m * p.N + n] = y;
          lo = fminf(lo, y);
          hi = fmaxf(hi, y);
        } else {
          reinterpret_cast<uint8_t *>(p.Y)[m * p.N + n] = (uint8_t)epi_requant(e, sc, v, n);
        }
      }
    }
    __syncthreads(); // part[] is rewritten by the next group
  }
  if (warp == 0 && p.out_range && p.kind == OMCUDA_EPI_DEQUANT)
    range_commit_warp(p.out_range, lo, hi);
}

// ---- GEMV-shaped GEMM for 2..16 rows on mma.sync ---------------------------------
//
// With more than one row the dp4a work per weight byte of the kernel above
// starts to outgrow the weight read.  This kernel keeps the same shape (a pass over the weight,
// HBM bound) and hands the arithmetic to mma.sync.m16n8k32: the 16 rows of
// the A fragment are the (up to) 16 rows of the problem, the 8 columns of the
// B fragment are 8 adjacent output columns, and a warp consumes the weight in
// 64-byte blocks of K: lane (g, q) (g = lane / 4 the column, q = lane % 4)
// loads the 16 bytes at offset 16 q of column g's block straight from global
// memory into its B registers.  The instruction's own K order is different
// (lane q holds K bytes 4q..4q+3 and 16+4q..16+4q+3), but a sum over K does not
// care in which order the bytes are paired as long as A and B agree, so A is
// loaded with the same permutation (the 16 bytes at offset 16 q of rows g and
// g + 8) and one 16-byte load feeds two MMAs.  The kGemvMmaWarps warps of a
// block split K between them and fold their fragments through shared memory;
// all threads then run the epilogue, consecutive threads on consecutive
// columns.  Integer sums are exact in any order: bit-identical to the other
// kernels.
constexpr int kGemvMmaWarps = 8;
constexpr int kGemvMmaUnroll = 4; // 64-byte blocks of K in flight per warp

template <int CG, bool kASigned, bool kBSigned>
__global__ void __launch_bounds__(32 * kGemvMmaWarps)
    gemm_i8_gemv_mma_kernel(const uint8_t *__restrict__ A,
        const uint8_t *__restrict__ Bt, int64_t kp, EpiParams p) {
  constexpr int kCols = 8 * CG;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  const int64_t m0 = (int64_t)blockIdx.y * 16;
  const bool vec_ok = ((p.lda & 15) == 0) && (((uintptr_t)A & 15u) == 0);
  const int64_t blocks64 = (kp + 63) >> 6;
  __shared__ int32_t part[kGemvMmaWarps][16][kCols + 1];
  __shared__ RangeBlock range;
  if (threadIdx.x == 0)
    range_block_init(range, kGemvMmaWarps); // (barriers follow: every block has a group)
  float lo = INFINITY, hi = -INFINITY;
  const int64_t groups = ceil_div(p.N, kCols);
  if (blockIdx.y == 0)
    for (int64_t grp = blockIdx.x; grp < groups; grp += gridDim.x)
      prefetch_weight(Bt, kp, grp * kCols, kCols, p.N);
  if (p.early_next)
    pdl_sync();
  else
    pdl_wait();
  A = after_pdl(A);
  Bt = after_pdl(Bt);
  const EpiScalars sc = epi_scalars(p);
  for (int64_t grp = blockIdx.x; grp < groups; grp += gridDim.x) {
    const int64_t n0 = grp * kCols;
    int32_t acc[CG][4];
#pragma unroll
    for (int j = 0; j < CG; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        acc[j][i] = 0;
    const uint8_t *brow[CG];
#pragma unroll
    for (int j = 0; j < CG; ++j) { // columns past N re-read the last one; never stored
      const int64_t n = n0 + 8 * j + g;
      brow[j] = Bt + (n < p.N ? n : p.N - 1) * kp + 16 * q;
    }
    // Warp w takes runs of kGemvMmaUnroll adjacent blocks (256 bytes of every
    // column), run r = w, w + kGemvMmaWarps, ...
    for (int64_t b0 = (int64_t)warp * kGemvMmaUnroll; b0 < blocks64;
         b0 += (int64_t)kGemvMmaWarps * kGemvMmaUnroll) {
      uint4 bw[kGemvMmaUnroll][CG];
#pragma unroll
      for (int u = 0; u < kGemvMmaUnroll; ++u) {
        const int64_t koff = ((b0 + u) << 6) + 16 * q;
#pragma unroll
        for (int j = 0; j < CG; ++j)
          bw[u][j] = koff < kp
                         ? __ldcs(reinterpret_cast<const uint4 *>(brow[j] + ((b0 + u) << 6)))
                         : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < kGemvMmaUnroll; ++u) {
        const int64_t koff = ((b0 + u) << 6) + 16 * q;
        const uint4 a_lo = load_a_chunk(A, m0 + g, p, koff, vec_ok);
        const uint4 a_hi = load_a_chunk(A, m0 + g + 8, p, koff, vec_ok);
#pragma unroll
        for (int j = 0; j < CG; ++j) {
          mma_m16n8k32<kASigned, kBSigned>(
              acc[j], a_lo.x, a_hi.x, a_lo.y, a_hi.y, bw[u][j].x, bw[u][j].y);
          mma_m16n8k32<kASigned, kBSigned>(
              acc[j], a_lo.z, a_hi.z, a_lo.w, a_hi.w, bw[u][j].z, bw[u][j].w);
        }
      }
    }
    // Accumulator fragment: c0,c1 = row g, columns 2q, 2q+1; c2,c3 = row g + 8.
#pragma unroll
    for (int j = 0; j < CG; ++j) {
      part[warp][g][8 * j + 2 * q] = acc[j][0];
      part[warp][g][8 * j + 2 * q + 1] = acc[j][1];
      part[warp][g + 8][8 * j + 2 * q] = acc[j][2];
      part[warp][g + 8][8 * j + 2 * q + 1] = acc[j][3];
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < 16 * kCols; idx += 32 * kGemvMmaWarps) {
      const int r = idx / kCols, cidx = idx % kCols;
      const int64_t m = m0 + r, n = n0 + cidx;
      if (m < p.M && n < p.N) {
        int32_t sum = 0;
#pragma unroll
        for (int w = 0; w < kGemvMmaWarps; ++w)
          sum += part[w][r][cidx];
        const EpiParams e = epi_after_pdl(p);
        const EpiRow row = epi_row(e, m);
        const int32_t v = epi_int(e, row, sum, n);
        if (p.kind == OMCUDA_EPI_I32) {
          reinterpret_cast<int32_t *>(p.Y)[m * p.N + n] = v;
        } else if (p.kind == OMCUDA_EPI_DEQUANT) {
          float y = epi_dequant(e, sc, v, n);
          if (e.residual)
            y = __fadd_rn(y, __ldg(e.residual + m * p.N + n));
          reinterpret_cast<float *>(p.Y)[m * p.N + n] = y;
          lo = fminf(lo, y);
          hi = fmaxf(hi, y);
        } else {
          reinterpret_cast<uint8_t *>(p.Y)[m * p.N + n] = (uint8_t)epi_requant(e, sc, v, n);
        }
      }
    }
    __syncthreads(); // part[] is rewritten by the next group
  }
  if (p.out_range && p.kind == OMCUDA_EPI_DEQUANT)
    range_commit_block(range, p.out_range, lo, hi, blockIdx.y * gridDim.x + blockIdx.x);
}

EpiParams make_epi_params(const GemmCall &a) {
  EpiParams p;
  p.M = a.M;
  p.N = a.N;
  p.K = a.K;
  p.lda = a.lda;
  p.a_zp = a.a_zp;
  p.a_zp_len = a.a_zp ? (int)(a.a_zp_len > 1 ? 2 : a.a_zp_len) : 0;
  p.a_signed = a.a_signed;
  p.b_zp = a.b_zp;
  p.b_zp_len = a.b_zp ? (int)(a.b_zp_len > 1 ? 2 : a.b_zp_len) : 0;
  p.b_signed = a.B.b_signed;
  p.colsum = a.B.colsum;
  p.rowsum = a.a_rowsum;
  p.kind = a.epilogue;
  p.Y = a.Y;
  p.sa = a.sa;
  p.sb = a.sb;
  p.sb_len = a.sb_len > 1 ? 2 : (int)a.sb_len;
  p.form = a.scale_form;
  p.bias = a.bias;
  p.gelu = a.gelu;
  p.y_zp = a.y_zp;
  p.y_zp_dev = a.y_zp_dev;
  p.residual = (a.epilogue == OMCUDA_EPI_DEQUANT) ? a.residual : nullptr;
  p.res_vec_ok = ((((uintptr_t)a.residual) & 15u) == 0) && (a.N % 4 == 0);
  p.out_range = reinterpret_cast<uint32_t *>(a.out_minmax);
  p.q_range = reinterpret_cast<const uint32_t *>(a.q_range);
  p.q_params = a.q_params;
  p.q_scale = a.q_scale;
  p.q_zp = a.q_zp;
  // (a scalar scale is read with a scalar load wherever it lies)
  const uintptr_t sb_vec = a.sb_len > 1 ? (uintptr_t)a.sb : 0;
  p.vec_ok = ((((uintptr_t)a.B.colsum | (uintptr_t)a.bias | sb_vec) & 15u) == 0) &&
             (a.N % 4 == 0);
  p.l2_hints = 0;
  p.early_next = a.early_next;
  p.quant_mode = quant_mode();
  p.split_k = 1;
  p.ws_rows = 0;
  return p;
}

template <int MT>
static void launch_warp_gemm(const GemmCall &a, cudaStream_t st) {
  EpiParams p = make_epi_params(a);
  dim3 grid((unsigned)ceil_div(a.N, 8), (unsigned)ceil_div(a.M, MT));
  const uint8_t *A = (const uint8_t *)a.A;
  const uint8_t *Bt = (const uint8_t *)a.B.bt;
  int sel = (a.a_signed ? 2 : 0) | (a.B.b_signed ? 1 : 0);
  switch (sel) {
  case 0:
    gemm_i8_warp_kernel<MT, false, false><<<grid, 256, 0, st>>>(A, Bt, a.B.kp, p);
    break;
  case 1:
    gemm_i8_warp_kernel<MT, false, true><<<grid, 256, 0, st>>>(A, Bt, a.B.kp, p);
    break;
  case 2:
    gemm_i8_warp_kernel<MT, true, false><<<grid, 256, 0, st>>>(A, Bt, a.B.kp, p);
    break;
  default:
    gemm_i8_warp_kernel<MT, true, true><<<grid, 256, 0, st>>>(A, Bt, a.B.kp, p);
    break;
  }
}

// Warps per block for one row.  What a block does between its loads (the fold, the tail, the
// next group's addresses) leaves its warps without any in flight, and a launch that needs
// several groups per block repeats that; short blocks that all fit at once overlap it.  So
// the most warps for which every group of columns has a resident block, no more than have
// work on a short K, and eight only where no more than two threads in seven sit out the last
// trip.  us a call, weights beyond L2, with 8 / 4 / 2 / 1 warps:
//   K x N      3000 x 768  6.1 / 6.5 / 6.7 / 7.7      11008 x 1536   9.3 / 10.2 / 11.3 / 15.4
//              5500 x 1536 7.7 / 7.6 / 8.6 / 9.6       2048 x 768    5.9 / 5.8 / 6.1 / 6.8
//              4096 x 4096 10.1 / 8.7 / 9.1 / 10.3     4096 x 6144  12.2 / 10.6 / 9.9 / 10.3
//              4096 x 14336 21.1 / 16.1 / 14.9 / 13.9  1024 x 50000 42.8 / 23.6 / 16.5 / 13.2
//              8192 x 20000 32.2 / 30.1 / 30.7 / 31.6
static int gemv_warps(int64_t N, int64_t kp) {
  const int64_t groups = ceil_div(N, 4), sms = sm_count(), chunks = kp >> 4;
  if (groups <= 3 * sms && ceil_div(chunks, 256) * 256 * 5 <= chunks * 7)
    return 8;
  if (chunks > 64 && groups <= 8 * sms)
    return 4;
  return groups <= 16 * sms ? 2 : 1;
}

template <int MT, int CB, int kWarps>
static void launch_gemv(const GemmCall &a, cudaStream_t st) {
  EpiParams p = make_epi_params(a);
  // As many blocks as are resident together (64 registers a thread; 8 x 16-byte loads in
  // flight each with CB = 4), each with the same number of column groups, give or take one.
  // (A grid for twelve blocks of four warps, of which eight fit, ran a second round for the
  // last: 1 x 4096 x 14336 19.2 us a call, 16.1 with eight.)
  const int64_t groups = ceil_div(a.N, CB);
  const int64_t resident = (int64_t)sm_count() * (kGemvSmWarps / kWarps);
  const int64_t rounds = ceil_div(groups, resident);
  dim3 grid((unsigned)ceil_div(groups, rounds), (unsigned)ceil_div(a.M, MT));
  const uint8_t *A = (const uint8_t *)a.A;
  const uint8_t *Bt = (const uint8_t *)a.B.bt;
  const int threads = 32 * kWarps;
  int sel = (a.a_signed ? 2 : 0) | (a.B.b_signed ? 1 : 0);
  switch (sel) {
  case 0:
    (void)launch_pdl(
        gemm_i8_gemv_kernel<MT, CB, kWarps, false, false>, grid, threads, 0, st, 0, true, A, Bt, a.B.kp, p);
    break;
  case 1:
    (void)launch_pdl(
        gemm_i8_gemv_kernel<MT, CB, kWarps, false, true>, grid, threads, 0, st, 0, true, A, Bt, a.B.kp, p);
    break;
  case 2:
    (void)launch_pdl(
        gemm_i8_gemv_kernel<MT, CB, kWarps, true, false>, grid, threads, 0, st, 0, true, A, Bt, a.B.kp, p);
    break;
  default:
    (void)launch_pdl(
        gemm_i8_gemv_kernel<MT, CB, kWarps, true, true>, grid, threads, 0, st, 0, true, A, Bt, a.B.kp, p);
    break;
  }
}

template <int CG>
static void launch_gemv_mma(const GemmCall &a, cudaStream_t st) {
  EpiParams p = make_epi_params(a);
  // One block per 8 * CG columns (it reads 8 * CG * K bytes of the weight); very
  // wide weights wrap around a grid of 16 blocks per SM.
  const int64_t groups = ceil_div(a.N, 8 * CG), cap = (int64_t)sm_count() * 16;
  dim3 grid((unsigned)(groups < cap ? groups : cap), (unsigned)ceil_div(a.M, 16));
  const uint8_t *A = (const uint8_t *)a.A;
  const uint8_t *Bt = (const uint8_t *)a.B.bt;
  const int threads = 32 * kGemvMmaWarps;
  int sel = (a.a_signed ? 2 : 0) | (a.B.b_signed ? 1 : 0);
  switch (sel) {
  case 0:
    (void)launch_pdl(
        gemm_i8_gemv_mma_kernel<CG, false, false>, grid, threads, 0, st, 0, true, A, Bt, a.B.kp, p);
    break;
  case 1:
    (void)launch_pdl(
        gemm_i8_gemv_mma_kernel<CG, false, true>, grid, threads, 0, st, 0, true, A, Bt, a.B.kp, p);
    break;
  case 2:
    (void)launch_pdl(
        gemm_i8_gemv_mma_kernel<CG, true, false>, grid, threads, 0, st, 0, true, A, Bt, a.B.kp, p);
    break;
  default:
    (void)launch_pdl(
        gemm_i8_gemv_mma_kernel<CG, true, true>, grid, threads, 0, st, 0, true, A, Bt, a.B.kp, p);
    break;
  }
}

// OMCUDA_GEMV=0 keeps the older warp-per-column kernel for every M, for
// experiments.
static bool gemv_wanted() {
  static const bool on = [] {
    const char *s = getenv("OMCUDA_GEMV");
    return !(s && atoi(s) == 0);
  }();
  return on;
}

// Largest M the mma.sync GEMV takes (row groups of 16 re-read the weight
// through L2).  OMCUDA_GEMV_MMA_MAX_M overrides it; 0 switches the kernel off.
static int64_t gemv_mma_max_m() {
  static const int64_t v = [] {
    const char *s = getenv("OMCUDA_GEMV_MMA_MAX_M");
    return s ? (int64_t)atoll(s) : (int64_t)16;
  }();
  return v;
}

static int64_t gemv_max_m() {
  if (!gemv_wanted())
    return 0;
  return gemv_mma_max_m() > 4 ? gemv_mma_max_m() : 4;
}

int launch_gemm_simt(const GemmCall &a, cudaStream_t st) {
  // The GEMV-shaped kernels: dp4a up to 4 rows, mma.sync above (with more
  // rows the dp4a work per weight byte outgrows the weight read).
  // (OMCUDA_GEMV_MMA_MIN_M moves the hand-over from the dp4a kernel, for
  // experiments: measured on 4096 x 14336 the dp4a kernel reads one row's
  // weight in 19 us, 14 with shorter blocks, and four rows' in 29 us, the mma.sync kernel 22
  // and 24 us.)
  static const int64_t mma_min_m = [] {
    const char *s = getenv("OMCUDA_GEMV_MMA_MIN_M");
    return s ? (int64_t)atoll(s) : (int64_t)2;
  }();
  if (a.M >= mma_min_m && a.M <= gemv_mma_max_m() && gemv_wanted()) {
    launch_gemv_mma<2>(a, st);
    OMCUDA_CHECK_LAUNCH("gemm_i8_gemv_mma_kernel");
    return OMCUDA_OK;
  }
  if (a.M <= 16 && gemv_wanted()) {
    if (a.M <= 1)
      switch (gemv_warps(a.N, a.B.kp)) {
      case 1:
        launch_gemv<1, 4, 1>(a, st);
        break;
      case 2:
        launch_gemv<1, 4, 2>(a, st);
        break;
      case 4:
        launch_gemv<1, 4, 4>(a, st);
        break;
      default:
        launch_gemv<1, 4, 8>(a, st);
      }
    else if (a.M <= 2)
      launch_gemv<2, 4, 4>(a, st);
    else if (a.M <= 4)
      launch_gemv<4, 4, 4>(a, st);
    else
      launch_gemv<8, 4, 4>(a, st); // 9..16 rows: two row groups share the weight through L2
    OMCUDA_CHECK_LAUNCH("gemm_i8_gemv_kernel");
    return OMCUDA_OK;
  }
  if (a.M <= 1)
    launch_warp_gemm<1>(a, st);
  else if (a.M <= 4)
    launch_warp_gemm<4>(a, st);
  else if (a.M <= 8)
    launch_warp_gemm<8>(a, st);
  else
    launch_warp_gemm<16>(a, st);
  OMCUDA_CHECK_LAUNCH("gemm_i8_warp_kernel");
  return OMCUDA_OK;
}

namespace {

// Shared memory that rowsum_kernel does not use, but that keeps its blocks apart when
// they copy rows.  Set up behind a tensor-core kernel, the blocks go to the SMs that
// kernel leaves idle, up to eight to an SM, and the copy then runs on those alone:
// MatMulInteger 1024 x 4008 x 1024, whose tiles leave 20 SMs, 20.6 us without the
// overlap, 22.2 with it, 19.7 with two blocks to an SM; 512 x 9000 x 1024 24.6, 22.7
// and 22.2.  Four to an SM where the grid has them (4096 x 4008 x 1024 28.7, 28.0, 27.3).
constexpr size_t kSpreadTwo = 100 * 1024, kSpreadFour = 48 * 1024;
size_t spread_smem(int64_t blocks) {
  static PerDeviceInt cached; // 1: two to an SM can be asked for, 2: not
  int can = cached.get();
  if (can == 0) {
    const bool ok = cudaFuncSetAttribute(rowsum_kernel<true>,
                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSpreadTwo) ==
                        cudaSuccess &&
                    cudaFuncSetAttribute(rowsum_kernel<false>,
                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSpreadTwo) ==
                        cudaSuccess;
    (void)cudaGetLastError();
    can = ok ? 1 : 2;
    cached.set(can);
  }
  const int64_t per_sm = ceil_div(blocks, (int64_t)sm_count());
  return per_sm <= 2 && can == 1 ? kSpreadTwo : per_sm <= 4 ? kSpreadFour : 0;
}

} // namespace

int launch_repitch(const void *A, int a_signed, int64_t M, int64_t K, int64_t pitch,
    uint8_t *dst, int32_t *rowsum, const RequantScale &rq, cudaStream_t st, const void *zp,
    int64_t zp_len) {
  const int64_t blocks = ceil_div(M, 8) + ceil_div(rq.len, 256);
  // (a block's rows are 8 K bytes: more zero points than that cost more than they save)
  const uint8_t *look = zp_len <= 8 * K ? (const uint8_t *)zp : nullptr;
  const bool overlap = pdl_pays(M * K);
  const size_t spread = dst && overlap ? spread_smem(blocks) : 0;
  OMCUDA_CHECK(launch_pdl(a_signed ? rowsum_kernel<true> : rowsum_kernel<false>,
      (unsigned)blocks, 256, spread, st, 0, overlap, (const uint8_t *)A, M, K, rowsum, dst,
      pitch, look, zp_len, rq));
  OMCUDA_CHECK_LAUNCH("rowsum_kernel");
  return OMCUDA_OK;
}

} // namespace omcuda

using namespace omcuda;

extern "C" int64_t omcudaDevPreparedBBytes(int64_t K, int64_t N, int64_t *kp) {
  int64_t k16 = (K + 15) & ~int64_t(15);
  if (kp)
    *kp = k16;
  return N * k16;
}

extern "C" int omcudaDevPrepareB(const void *B, int b_signed, int64_t K,
    int64_t N, omcudaPreparedB *out, void *stream) {
  if (!B || !out || !out->bt || !out->colsum || K <= 0 || N <= 0)
    return fail(OMCUDA_EINVAL, "PrepareB: bad argument");
  cudaStream_t st = (cudaStream_t)stream;
  int64_t kp;
  omcudaDevPreparedBBytes(K, N, &kp);
  out->K = K;
  out->N = N;
  out->kp = kp;
  out->b_signed = b_signed;
  dim3 tgrid((unsigned)ceil_div(N, 64), (unsigned)ceil_div(kp, 64));
  transpose_b_kernel<<<tgrid, 256, 0, st>>>(
      (const uint8_t *)B, K, N, kp, (uint8_t *)out->bt);
  OMCUDA_CHECK_LAUNCH("transpose_b_kernel");
  // Column sums of B are row sums of its copy (whose padding is zero): coalesced
  // 16-byte loads of what has just been written, on the whole machine.  (Last, and it
  // does not write the copy: whoever is launched behind it with overlap may start once it has.)
  return launch_repitch(out->bt, b_signed, N, kp, 0, nullptr, out->colsum, RequantScale(), st);
}

extern "C" int omcudaDevRowSum(const void *A, int a_signed, int64_t M,
    int64_t K, int32_t *rowsum, void *stream) {
  if (!A || !rowsum || M <= 0 || K <= 0)
    return fail(OMCUDA_EINVAL, "RowSum: bad argument");
  cudaStream_t st = (cudaStream_t)stream;
  return launch_repitch(A, a_signed, M, K, 0, nullptr, rowsum, RequantScale(), st);
}

extern "C" int omcudaDevRequantScale(const float *a_scale, const float *b_scale,
    int64_t len, const float *y_scale, float *S, void *stream) {
  if (!a_scale || !b_scale || !y_scale || !S || len <= 0)
    return fail(OMCUDA_EINVAL, "RequantScale: bad argument");
  requant_scale_kernel<<<(unsigned)ceil_div(len, 256), 256, 0,
      (cudaStream_t)stream>>>(RequantScale{a_scale, b_scale, y_scale, len, S});
  OMCUDA_CHECK_LAUNCH("requant_scale_kernel");
  return OMCUDA_OK;
}

extern "C" int omcudaDevGemmI8(const omcudaGemmArgs *args, void *stream) {
  if (!args)
    return fail(OMCUDA_EINVAL, "GemmI8: null args");
  return gemm_i8(GemmCall(*args), (cudaStream_t)stream);
}

// Whether a product that the few-rows kernel can run goes there; otherwise it runs on the
// 128- and 256-row tiles (use_tc), which a switch may have asked for, or the kernels for
// at most 16 rows.
static bool few_takes(int64_t M, int64_t N, int64_t K, bool use_tc) {
  return gemm_few_wanted(M, N, K) && !(use_tc && gemm_tc_forced());
}

extern "C" int omcudaDevGemmFewPlan(int64_t M, int64_t N, int64_t K, int *rows, int *split) {
  if (M <= 0 || N <= 0 || K <= 0 || !rows || !split)
    return fail(OMCUDA_EINVAL, "GemmFewPlan: bad argument"), -1;
  *rows = *split = 0;
  if (!few_takes(M, N, K, M > gemv_max_m()))
    return 0;
  gemm_few_plan(M, N, K, rows, split);
  return 1;
}

int omcuda::gemm_i8(const GemmCall &a, cudaStream_t st) {
  if (a.M < 0 || a.N <= 0 || a.K <= 0 || !a.A || !a.B.bt ||
      (!a.Y && a.epilogue != OMCUDA_EPI_DEQUANT_RANGE))
    return fail(OMCUDA_EINVAL, "GemmI8: bad shape or null operand");
  if (a.M == 0)
    return OMCUDA_OK;
  if (a.B.K != a.K || a.B.N != a.N)
    return fail(OMCUDA_EINVAL, "GemmI8: prepared B does not match K,N");
  if (a.a_zp && a.a_zp_len != 1 && a.a_zp_len != a.M)
    return fail(OMCUDA_EINVAL, "GemmI8: a_zp length must be 1 or M");
  if (a.b_zp && a.b_zp_len != 1 && a.b_zp_len != a.N)
    return fail(OMCUDA_EINVAL, "GemmI8: b_zp length must be 1 or N");
  if (a.b_zp && a.b_zp_len != 0 && !a.a_rowsum)
    return fail(OMCUDA_EINVAL, "GemmI8: b_zp needs the row sums of A");
  if (a.a_zp && a.a_zp_len != 0 && !a.B.colsum)
    return fail(OMCUDA_EINVAL, "GemmI8: a_zp needs the column sums of B");
  if (a.residual && a.epilogue != OMCUDA_EPI_DEQUANT)
    return fail(OMCUDA_EINVAL, "GemmI8: a residual goes with the dequant epilogue only");
  if (a.epilogue < OMCUDA_EPI_I32 || a.epilogue > OMCUDA_EPI_DEQUANT_QUANT)
    return fail(OMCUDA_EINVAL, "GemmI8: unknown epilogue %d", a.epilogue);
  if (epi_is_dequant(a.epilogue) && (!a.sa || !a.sb))
    return fail(OMCUDA_EINVAL, "GemmI8: dequant epilogue needs both scales");
  if (a.epilogue == OMCUDA_EPI_DEQUANT_RANGE && !a.out_minmax)
    return fail(OMCUDA_EINVAL, "GemmI8: the range-only tail needs out_minmax");
  if (a.epilogue == OMCUDA_EPI_DEQUANT_QUANT && (!a.q_range || !a.q_params))
    return fail(OMCUDA_EINVAL, "GemmI8: the quantizing tail needs q_range and q_params");
  if (a.epilogue == OMCUDA_EPI_REQUANT && !a.sb)
    return fail(OMCUDA_EINVAL, "GemmI8: requant epilogue needs S");
  if (a.epilogue != OMCUDA_EPI_I32 && a.sb_len != 1 && a.sb_len != a.N)
    return fail(OMCUDA_EINVAL, "GemmI8: scale length must be 1 or N");
  bool tc_ok = gemm_tc_supported(a);
  if (a.kernel_choice == 1 && !tc_ok)
    return fail(OMCUDA_ENOTSUP,
        "GemmI8: the tensor-core kernel needs 16-byte aligned rows of A");
  const bool tc_only = a.epilogue == OMCUDA_EPI_DEQUANT_SPLIT ||
                       a.epilogue == OMCUDA_EPI_DEQUANT_RANGE ||
                       a.epilogue == OMCUDA_EPI_DEQUANT_QUANT;
  if (tc_only && (!tc_ok || a.kernel_choice == 2))
    return fail(OMCUDA_ENOTSUP,
        "GemmI8: the split-bf16, range-only and quantizing tails exist on the "
        "tensor-core kernel only (16-byte aligned rows of A)");
  // With a handful of rows the GEMM is one read of the weight, which the
  // GEMV-shaped kernels stream faster than 128-row tensor-core tiles on a few
  // SMs (a row by 4096 x 14336: 14 us, on the few-rows kernel 15.3, on 128-row tiles 23-27).
  const bool use_tc = (a.kernel_choice == 1) || tc_only ||
                      (a.kernel_choice == 0 && tc_ok && a.M > gemv_max_m());
  if (a.kernel_choice == 0 && gemm_few_supported(a) && few_takes(a.M, a.N, a.K, use_tc))
    return launch_gemm_few(a, st);
  return use_tc ? launch_gemm_tc(a, st) : launch_gemm_simt(a, st);
}
