// Attention on the Blackwell tensor cores (tcgen05.mma kind::f16, bf16
// operands, fp32 accumulators in tensor memory) for the encoder graphs:
// softmax(Q K^T * scale) V per (batch, head), head size 64, sequence length a
// multiple of 128.
//
// It stands for the chain the reference lowers with CPU loops: two batched
// fp32 MatMuls (src/Conversion/ONNXToKrnl/Math/MatMul.cpp:488-507), a Mul by a
// constant and a Softmax over the last axis
// (src/Conversion/ONNXToKrnl/Math/Softmax.cpp:25-134).
//
// Accuracy.  Every fp32 operand a arrives already split as a = hi + lo with
// hi = bf16(a), lo = bf16(a - hi) (two bf16 planes, written by the QKV GEMM's
// epilogue or by split_bf16_kernel below), and each product is evaluated as
// lo*hi + hi*lo + hi*hi, which leaves a relative error of about 2^-16 per
// product, far inside the 1e-3 tolerance of the fp32 ops; accumulation is
// fp32.  The softmax runs online over key blocks (an exponent offset that
// tracks the running maximum, and the running sum), the same function as the
// reference's three-loop form up to fp32 rounding.
//
// Layout in HBM: the planes are [T, ld] bf16 row-major (T = batch*seq tokens);
// head h of Q / K / V owns columns [col + 64 h, col + 64 h + 64) of its rows.
// out is [T, ld_out] fp32.
//
// A work item = 128 query rows of one (batch, head).  Two persistent CTAs
// share an SM, so that one's softmax (CUDA cores) overlaps the other's matrix
// products (tensor pipe); each walks its share of the items.  Per block of 128
// keys:
//   the product warp (att_products) issues S = Q K^T as 12 MMAs (3 split terms
//              x 4 k-steps) into tensor memory;
//   8 warps    two threads per query row (its TMEM lane), 64 keys each: row
//              maximum (exchanged through shared memory), p = 2^(s*c - m),
//              running sum, p split into bf16 hi/lo and stored back over the
//              scores in tensor memory;
//   the product warp issues O_j = P V as 24 MMAs with P read from tensor memory
//              and V (keys x 64, MN-major) from shared memory: per 16-key
//              slice P_hi V_hi and P_lo V_hi into 64 columns of tensor memory,
//              P_hi V_lo into 64 others; and once they are done the next
//              block's S;
//   the load warp (att_loads) refills each buffer (TMA, 128-byte swizzle) once
//              the products that read it are done, and sends results off.
// O accumulates in tensor memory over the key blocks of an item (the P V MMAs
// add to it); the exponent offset of a row follows its running maximum lazily,
// moving only when a block's maximum exceeds it by more than 2^8, and only
// then are O and the row sum rescaled (a tensor-memory load / multiply /
// store pass): on typical data one pass or none per item instead of one
// register fold per block.  At the end of the item the 8 warps read O (the sum
// of its two 64-column halves), normalise and stage it in shared memory, from
// which it leaves with two TMA stores of whole 128-byte lines.
//
// What bounds it: the chain of a CTA (scores -> softmax -> P V -> scores), two of
// which share an SM.  One warp used to issue products and copies beside its rows,
// with a CTA barrier between any two phases: of some 5100 clocks per block 1180 were
// spent issuing copies and waking up, and 2600 more per item on its results.  Now warps
// of their own issue products and copies, mbarriers stand between the phases and the
// results are out of V's way (two CTAs share the SM: the tensor pipe counts 1536 clocks per block and CTA).
// Batch x sequence x heads, us: 256 x 512 x 16 829 -> 741, 64 x 384 x 16 124 -> 113, 1 x 512 x
// 16 13.8 -> 12.4, 32 x 128 x 12 11.6 -> 11.5, 1024 x 128 x 16 336 -> 325 (HBM).  The largest runs
// at the power limit, clocks at 1.35 GHz.  Every sum is in the order it was in.
// Every wait on an mbarrier is bounded (tc_ptx.cuh); a timeout raises the
// CTA's abort flag, the CTA frees its tensor memory, writes the status word
// and returns.
#include <cuda_bf16.h>

#include <cstdlib>
#include <cstring>

#include "../common.cuh"
#include "../runtime/internal.h"
#include "tc_ptx.cuh"

namespace omcuda {

namespace {

constexpr int kTQ = 128;            // query rows per CTA
constexpr int kTK = 128;            // keys per block
constexpr int kTDh = 64;            // head size
constexpr int kTile = 128 * 128;    // bytes of one 128-row x 64-bf16 tile
constexpr int kTcAttSmem = 6 * kTile + 1024;
constexpr uint32_t kTmemColsAtt = 256; // S/P: 0..127, O_j: 128..255
constexpr int kTcAttWarps = 8;         // two threads per query row
constexpr int kTcAttThreads = 32 * kTcAttWarps + 64; // and the two warps that feed them

// S = Q K^T of a block: twelve MMAs over the four 16-element K slices (32 bytes,
// descriptor + 2) of three pairs of operands, small terms first: Ql Kh, Qh Kl, Qh Kh.
// In one asm block, all descriptors made before the first: what the lone issuing thread
// does between two tcgen05.mma delays the next by some 100 cycles, during which the
// tensor pipe has nothing to do.  (Issued by an elected lane, that is little: as three
// blocks of four, and P V as four, encoder base 32 x 128 1403 us and 1404 so, large 256 x
// 512 97.5 and 95.6 ms where runs differ by 1.3 %.)
__device__ __forceinline__ void umma_scores(uint32_t d_tmem, uint64_t ql, uint64_t qh,
    uint64_t kh, uint64_t kl, uint32_t idesc) {
  asm volatile("{\n\t"
               ".reg .pred f, t;\n\t"
               ".reg .b64 ql1, ql2, ql3, qh1, qh2, qh3, kh1, kh2, kh3, kl1, kl2, kl3;\n\t"
               "setp.ne.b32 f, 0, 0;\n\t"
               "setp.eq.b32 t, 0, 0;\n\t"
               "add.u64 ql1, %1, 2; add.u64 ql2, %1, 4; add.u64 ql3, %1, 6;\n\t"
               "add.u64 qh1, %2, 2; add.u64 qh2, %2, 4; add.u64 qh3, %2, 6;\n\t"
               "add.u64 kh1, %3, 2; add.u64 kh2, %3, 4; add.u64 kh3, %3, 6;\n\t"
               "add.u64 kl1, %4, 2; add.u64 kl2, %4, 4; add.u64 kl3, %4, 6;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %3, %5, f;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], ql1, kh1, %5, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], ql2, kh2, %5, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], ql3, kh3, %5, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %2, %4, %5, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], qh1, kl1, %5, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], qh2, kl2, %5, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], qh3, kl3, %5, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %2, %3, %5, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], qh1, kh1, %5, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], qh2, kh2, %5, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], qh3, kh3, %5, t;\n\t"
               "}" ::"r"(d_tmem),
               "l"(ql), "l"(qh), "l"(kh), "l"(kl), "r"(idesc)
               : "memory");
}

// O += P V of a block, 24 MMAs of 16 keys: A (P) from tensor memory, eight columns per slice,
// hi parts of 32 keys at column 0 and lo parts at 16 of every 32; B (V, MN-major) advances 16
// keys = 2048 bytes (descriptor + 128).  P_hi V_hi, then P_lo V_hi into columns 0..63, P_hi V_lo
// into 64..127.  All of one shape, for only products of one accumulator and one shape are promised
// to run in the order of issue (PTX ISA, pipelined tcgen05 instructions).  P_hi [V_hi | V_lo] as
// eight products of N = 128 with P_lo V_hi on top takes the tensor pipe as long (32 clocks per
// product of N = 64, 64 per one of N = 128) and was no faster: 64 x 384 x 16 114.2 and so 112.9 us,
// 16 x 512 x 16 54.7 and 53.1, 32 x 128 x 12 11.5 and 11.4, 1 x 512 x 16 11.9 and 11.9.
__device__ __forceinline__ void umma_values(uint32_t d_tmem, uint32_t p_tmem, uint64_t vl,
    uint64_t vh, uint32_t idesc, uint32_t accumulate_first) {
  asm volatile("{\n\t"
               ".reg .pred p, t;\n\t"
               ".reg .b32 a1, a2, a3, a4, a5, a6, a7, c0, c1, c2, c3, c4, c5, c6, c7, d1;\n\t"
               ".reg .b64 v1, v2, v3, v4, v5, v6, v7, w1, w2, w3, w4, w5, w6, w7;\n\t"
               "setp.ne.b32 p, %5, 0;\n\t"
               "setp.eq.b32 t, 0, 0;\n\t"
               "add.u32 d1, %0, 64;\n\t"
               "add.u32 a1, %1, 8; add.u32 a2, %1, 32; add.u32 a3, %1, 40; add.u32 a4, %1, 64;\n\t"
               "add.u32 a5, %1, 72; add.u32 a6, %1, 96; add.u32 a7, %1, 104;\n\t"
               "add.u32 c0, %1, 16; add.u32 c1, %1, 24; add.u32 c2, %1, 48; add.u32 c3, %1, 56;\n\t"
               "add.u32 c4, %1, 80; add.u32 c5, %1, 88; add.u32 c6, %1, 112; add.u32 c7, %1, 120;\n\t"
               "add.u64 v1, %2, 128; add.u64 v2, %2, 256; add.u64 v3, %2, 384; add.u64 v4, %2, 512;\n\t"
               "add.u64 v5, %2, 640; add.u64 v6, %2, 768; add.u64 v7, %2, 896;\n\t"
               "add.u64 w1, %3, 128; add.u64 w2, %3, 256; add.u64 w3, %3, 384; add.u64 w4, %3, 512;\n\t"
               "add.u64 w5, %3, 640; add.u64 w6, %3, 768; add.u64 w7, %3, 896;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %3, %4, p;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], w1, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], w2, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], w3, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [a4], w4, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [a5], w5, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [a6], w6, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [a7], w7, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [c0], %3, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [c1], w1, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [c2], w2, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [c3], w3, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [c4], w4, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [c5], w5, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [c6], w6, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [c7], w7, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [d1], [%1], %2, %4, p;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [d1], [a1], v1, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [d1], [a2], v2, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [d1], [a3], v3, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [d1], [a4], v4, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [d1], [a5], v5, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [d1], [a6], v6, %4, t;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [d1], [a7], v7, %4, t;\n\t"
               "}" ::"r"(d_tmem),
               "r"(p_tmem), "l"(vl), "l"(vh), "r"(idesc), "r"(accumulate_first)
               : "memory");
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(
          taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
      "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]),
      "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// {hi(b), hi(a)} as packed bf16 (a in the low half), round to nearest even.
__device__ __forceinline__ uint32_t cvt_bf16x2(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}

// Barrier between the two warps (64 threads) that share a lane quadrant;
// named barriers 1..4, constant ids so that only those are reserved.
__device__ __forceinline__ void pair_barrier(int quad) {
  switch (quad) {
  case 0:
    asm volatile("bar.sync 1, 64;" ::: "memory");
    break;
  case 1:
    asm volatile("bar.sync 2, 64;" ::: "memory");
    break;
  case 2:
    asm volatile("bar.sync 3, 64;" ::: "memory");
    break;
  default:
    asm volatile("bar.sync 4, 64;" ::: "memory");
    break;
  }
}

// Instruction descriptor of tcgen05.mma kind::f16 with bf16 operands and an
// fp32 accumulator, M = 128; b_mn_major selects an MN-major (transposed) B.
__host__ __device__ constexpr uint32_t att_idesc(int n, int b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)b_mn_major << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// Coordinates of one work item: 128 query rows of one (batch, head).
struct AttItem {
  int32_t row_q, row_kv, cq, ck, cv, col_out;
};

// Shared-memory addresses of the operand tiles, and of the mbarriers: tiles loaded (q, k, v),
// scores ready (s), P in tensor memory (p), P V done (o), results staged (r), and one for a CTA
// that gives up.
struct AttTiles {
  uint32_t qh, ql, kh, kl, vh, vl;
};
struct AttBars {
  uint32_t q, k, v, s, p, o, r, end;
};
struct AttLoads { // requested so far
  uint32_t q, k, v;
};

__device__ __forceinline__ AttItem att_item(int64_t item, int nq, int64_t S,
    int64_t heads, int32_t q_col, int32_t k_col, int32_t v_col) {
  const int64_t bh = item / nq, qt = item % nq;
  const int64_t b = bh / heads, h = bh % heads;
  AttItem it;
  it.row_kv = (int32_t)(b * S);
  it.row_q = it.row_kv + (int32_t)qt * kTQ;
  it.col_out = (int32_t)h * kTDh;
  it.cq = q_col + it.col_out;
  it.ck = k_col + it.col_out;
  it.cv = v_col + it.col_out;
  return it;
}

// For the product warp, whose wait is part of the chain: polls without being suspended for
// the first 4096 (mbarrier.try_wait wakes up some 100 clocks late: 1 x 512 x 16 14.9 -> 13.1 us,
// 256 x 512 x 16 746 -> 750), then waits like the others.
__device__ __forceinline__ bool mbar_spin(
    uint32_t bar, uint32_t parity, volatile int *abort_flag, uint64_t limit_ns) {
  for (int i = 0; i < 4096; ++i)
    if (mbar_test_wait(bar, parity))
      return true;
  return mbar_wait(bar, parity, abort_flag, limit_ns);
}

// The tensor pipe's part, by one elected thread of a warp that does nothing else.  Returns
// false when a wait ran out (or the CTA is aborting).
//
// The next block's S = Q K^T overwrites the columns that P V reads P from, and the two have
// different accumulators, whose order nothing promises (see umma_values): it waits for P V.
// (Queued right behind it, some 130 clocks a block less where a CTA has the SM for itself: 1 x
// 2048 x 9 heads 37.5 and so 39.6 us, 1 x 512 x 16 11.9 and 12.4; nothing measurable where two share
// it.)  With that, whoever has seen scores ready has seen every P V before them done as well.  The
// first block of the next item runs while the softmax warps are still busy with the results of the
// one before.
__device__ __forceinline__ bool att_products(const AttTiles &s, const AttBars &bar,
    uint32_t tmem, int nkb, int64_t n_items, volatile int *abortp, uint64_t wait_ns) {
  constexpr uint32_t kIdescQK = att_idesc(kTK, 0);
  constexpr uint32_t kIdescPV = att_idesc(kTDh, 1);
  static_assert(kTDh == 64, "four K slices per operand row");
  static_assert(kTK == 128, "eight 16-key slices per block");
  const uint32_t t_s = tmem, t_o = tmem + 128u;
  const uint64_t dqh = make_smem_desc(s.qh), dql = make_smem_desc(s.ql),
                 dkh = make_smem_desc(s.kh), dkl = make_smem_desc(s.kl),
                 dvh = make_smem_desc(s.vh), dvl = make_smem_desc(s.vl);
  auto wait = [&](uint32_t b, uint32_t parity) {
    return mbar_spin(b, parity & 1u, abortp, wait_ns);
  };
  uint32_t n = 0;     // key blocks, parity of bar.k / v / s / p / o
  uint32_t nitem = 0; // items, parity of bar.q
  if (!wait(bar.q, 0) || !wait(bar.k, 0))
    return false;
  tcgen05_fence_after();
  umma_scores(t_s, dql, dqh, dkh, dkl, kIdescQK);
  umma_commit(bar.s);
  for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x, ++nitem) {
    const bool has_next = item + gridDim.x < n_items;
    for (int j = 0; j < nkb; ++j, ++n) {
      const bool last = j + 1 == nkb;
      if (!wait(bar.v, n) || !wait(bar.p, n))
        return false;
      tcgen05_fence_after();
      umma_values(t_o, t_s, dvl, dvh, kIdescPV, j != 0 ? 1u : 0u);
      umma_commit(bar.o);
      if (!last || has_next) {
        if (!wait(bar.o, n) || (last && !wait(bar.q, nitem + 1)) || !wait(bar.k, n + 1))
          return false;
        tcgen05_fence_after();
        umma_scores(t_s, dql, dqh, dkh, dkl, kIdescQK);
        umma_commit(bar.s);
      }
    }
  }
  return true;
}

// The copies' part, by one elected thread of another warp: every buffer is refilled as soon as
// the products that read it are done.  loads: what it requested, for one that gives up.
__device__ __forceinline__ bool att_loads(const CUtensorMap &map_hi, const CUtensorMap &map_lo,
    const CUtensorMap &map_out, const AttTiles &s, const AttBars &bar, int32_t q_col,
    int32_t k_col, int32_t v_col, int nkb, int nq, int64_t S, int64_t heads, int64_t n_items,
    AttLoads &loads, volatile int *abortp, uint64_t wait_ns) {
  auto load = [&](uint32_t b, uint32_t hi, uint32_t lo, int32_t col, int32_t row) {
    mbar_expect_tx(b, 2 * kTile);
    tma_load_2d(hi, &map_hi, col, row, b);
    tma_load_2d(lo, &map_lo, col, row, b);
  };
  auto load_q = [&](const AttItem &it) {
    load(bar.q, s.qh, s.ql, it.cq, it.row_q), ++loads.q;
  };
  auto load_k = [&](const AttItem &it, int j) {
    load(bar.k, s.kh, s.kl, it.ck, it.row_kv + j * kTK), ++loads.k;
  };
  auto load_v = [&](const AttItem &it, int j) {
    load(bar.v, s.vh, s.vl, it.cv, it.row_kv + j * kTK), ++loads.v;
  };
  auto wait = [&](uint32_t b, uint32_t parity) {
    return mbar_wait(b, parity & 1u, abortp, wait_ns);
  };
  AttItem it = att_item(blockIdx.x, nq, S, heads, q_col, k_col, v_col);
  load_q(it);
  load_k(it, 0);
  load_v(it, 0);
  // The results of an item take a turn in the K buffers, once the next item's first scores are
  // done with them: the next K has the longest time to arrive.  Items of one key block have no
  // such next K; theirs take it in the V buffers.
  const bool in_v = nkb == 1;
  auto store = [&](const AttItem &at) {
    tma_store_2d(&map_out, in_v ? s.vh : s.kh, at.col_out, at.row_q);
    tma_store_2d(&map_out, in_v ? s.vl : s.kl, at.col_out + 32, at.row_q);
    tma_store_commit();
  };
  uint32_t n = 0, nitem = 0;
  AttItem before = it;
  for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x, ++nitem) {
    const bool has_next = item + gridDim.x < n_items;
    AttItem nx = it;
    if (has_next)
      nx = att_item(item + gridDim.x, nq, S, heads, q_col, k_col, v_col);
    for (int j = 0; j < nkb; ++j, ++n) {
      const bool last = j + 1 == nkb, more = !last || has_next;
      const AttItem &at = last ? nx : it; // of the next block
      const int jn = last ? 0 : j + 1;
      if (!wait(bar.s, n)) // the K buffers are free, behind an item's last block the Q buffers too
        return false;
      if (last && has_next)
        load_q(nx);
      if (j == 0 && nitem != 0 && !in_v) {
        if (!wait(bar.r, nitem - 1))
          return false;
        store(before);
        tma_store_wait_read();
      }
      if (more)
        load_k(at, jn);
      if (in_v) {
        if (!wait(bar.r, nitem))
          return false;
        store(it);
        tma_store_wait_read();
      } else if (more && !wait(bar.o, n)) {
        return false;
      }
      if (more)
        load_v(at, jn);
    }
    before = it;
    it = nx;
  }
  if (!in_v) {
    if (!wait(bar.r, nitem - 1))
      return false;
    store(before);
  }
  return true;
}

__global__ void __launch_bounds__(kTcAttThreads, 2)
    attention_tc_kernel(const __grid_constant__ CUtensorMap map_hi,
        const __grid_constant__ CUtensorMap map_lo,
        const __grid_constant__ CUtensorMap map_out, int32_t q_col, int32_t k_col,
        int32_t v_col, int64_t S, int64_t heads, int64_t n_items, float scale_log2e,
        uint32_t *__restrict__ out_range, int *status, uint64_t wait_ns) {
  extern __shared__ uint8_t att_tc_smem[];
  __shared__ uint64_t bars[8];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  // What the two threads of a row tell each other.  The maxima of a block lie where those of
  // the block before last did: a thread gets there past a barrier that its partner reaches
  // after having read them.  So do the sums, for there is a block between any two.
  __shared__ float xch_max[2][2][kTQ], xch_sum[2][kTQ];
  __shared__ RangeBlock range;

  const int tid = threadIdx.x, warp = warp_number(), lane = tid & 31;
  // Warps w and w + 4 share the 32 query rows (TMEM lanes) of quadrant w & 3:
  // `half` 0 takes keys 0..63 of every block and output columns 0..31, half 1
  // the rest.
  const int quad = warp & 3, half = warp >> 2;
  const int row = quad * 32 + lane;
  const int nkb = (int)(S / kTK);
  const int nq = (int)(S / kTQ);

  const uint32_t smem0 = (smem_u32(att_tc_smem) + 1023u) & ~1023u;
  const AttTiles tiles = {smem0, smem0 + kTile, smem0 + 2 * kTile, smem0 + 3 * kTile,
      smem0 + 4 * kTile, smem0 + 5 * kTile};
  const uint32_t bar0 = smem_u32(bars);
  const AttBars bar = {bar0, bar0 + 8, bar0 + 16, bar0 + 24, bar0 + 32, bar0 + 40, bar0 + 48,
      bar0 + 56};

  if (tid == 32) {
    prefetch_tensormap(&map_hi);
    prefetch_tensormap(&map_lo);
    prefetch_tensormap(&map_out);
  }
  if (tid == 0) {
    abort_flag = 0;
    range_block_init(range, kTcAttWarps);
    mbar_init(bar.q, 1);
    mbar_init(bar.k, 1);
    mbar_init(bar.v, 1);
    mbar_init(bar.s, 1);
    mbar_init(bar.p, kTcAttWarps);
    mbar_init(bar.o, 1);
    mbar_init(bar.r, kTcAttWarps);
    mbar_init(bar.end, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0)
    tmem_alloc(smem_u32(&tmem_slot), kTmemColsAtt);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_sync();
  volatile int *abortp = &abort_flag;

  // The CTA walks the items blockIdx.x, blockIdx.x + gridDim.x, ... (the grid has no more
  // CTAs than there are items).
  if (warp == kTcAttWarps) {
    if (elect_one() && !att_products(tiles, bar, tmem, nkb, n_items, abortp, wait_ns)) {
      // Gave up: tell the others, then let what is under way end before tensor memory goes.
      abort_flag = 1;
      volatile int own = 0;
      umma_commit(bar.end);
      (void)mbar_wait(bar.end, 0, &own, wait_ns);
    }
    __syncwarp();
  } else if (warp == kTcAttWarps + 1) {
    AttLoads loads = {0, 0, 0};
    const bool mine = elect_one();
    if (mine && !att_loads(map_hi, map_lo, map_out, tiles, bar, q_col, k_col, v_col, nkb, nq, S,
                           heads, n_items, loads, abortp, wait_ns)) {
      abort_flag = 1; // (as above, for the copies)
      const uint32_t b[3] = {bar.q, bar.k, bar.v}, asked[3] = {loads.q, loads.k, loads.v};
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        volatile int own = 0;
        (void)mbar_wait(b[i], (asked[i] - 1u) & 1u, &own, wait_ns);
      }
    }
    if (mine)
      tma_store_wait_all();
    __syncwarp();
  } else {
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    const uint32_t t_row = tmem + lane_base + (uint32_t)(half * (kTK / 2)); // its scores, then P
    const uint32_t t_out = tmem + 128u + lane_base + (uint32_t)(32 * half); // its part of O
    // A warp whose wait ran out goes on to the end all the same, with whatever tensor memory
    // holds: its partner meets it at every barrier of the pair, and the waits that follow end
    // as soon as they see the flag.
    bool ok = true;
    uint32_t n = 0;                              // key blocks
    float lo_run = INFINITY, hi_run = -INFINITY; // range of this thread's outputs

    for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x) {
      // O accumulates in tensor memory over the key blocks of the item.  The
      // exponent offset m_ref of a row follows its running maximum lazily: it
      // moves (and O and the row sum are rescaled) only when a block's maximum
      // exceeds it by more than 2^8, so p never exceeds 256 and most blocks
      // need no pass over O at all.  Any offset gives the same softmax once
      // the sum over the same p normalises the result.
      float m_ref = -INFINITY; // exponent offset, in units of s * scale * log2(e)
      float l_run = 0.0f;      // running sum of p

      for (int j = 0; j < nkb; ++j, ++n) {
        // (S is issued once P V of the block before is done, so bar.o is at most one phase behind
        // here and the wait for it at the end of the item may skip the phases between)
        ok = mbar_wait(bar.s, n & 1u, abortp, wait_ns) && ok;
        tcgen05_fence_after();

        // ---- online softmax: this thread's half of its row ----
        __syncwarp(); // tcgen05.ld / st are warp-collective: enter them converged
        // The thread's 64 scores are read from tensor memory once and stay in
        // registers for both passes (maximum, then exponentials).
        static_assert(kTK / 2 == 64, "two 32-column loads per thread");
        uint32_t sv[2][32];
        tmem_ld32(t_row, sv[0]);
        tmem_ld32(t_row + 32u, sv[1]);
        tmem_ld_wait();
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}; // (no chain of 32)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int i = 0; i < 32; i += 2)
            m4[(i >> 1) & 3] = max3f(m4[(i >> 1) & 3], __uint_as_float(sv[h][i]),
                __uint_as_float(sv[h][i + 1]));
        float mx = max3f(m4[0], m4[1], fmaxf(m4[2], m4[3]));
        // Row maximum over both halves (a named barrier per quadrant).
        xch_max[n & 1u][half][row] = mx;
        pair_barrier(quad);
        mx = fmaxf(mx, xch_max[n & 1u][half ^ 1][row]);
        const float m_blk = __fmul_rn(mx, scale_log2e);
        // (true for every row on the first block: m_ref is -inf)
        const bool move = m_blk > __fadd_rn(m_ref, 8.0f);
        // Both threads of a row and both warps of a quadrant see the same rows
        // and maxima, so they take this branch together.
        if (j > 0 && __any_sync(0xffffffffu, move)) {
          const float f = move ? ex2_approx(__fsub_rn(m_ref, m_blk)) : 1.0f;
          l_run = __fmul_rn(l_run, f);
          const uint64_t f2 = pack_f32x2(f, f);
#pragma unroll 1
          for (uint32_t part = 0; part < 4; ++part) { // P_hi V_hi + P_lo V_hi | P_hi V_lo
            const uint32_t ta = t_out + (part >> 1) * 64u + (part & 1u) * 16u;
            uint32_t v[16];
            tmem_ld16(ta, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              float a, b;
              unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), f2), a, b);
              v[i] = __float_as_uint(a);
              v[i + 1] = __float_as_uint(b);
            }
            tmem_st16(ta, v);
          }
          tmem_st_wait();
        }
        if (move)
          m_ref = m_blk;
        // (packed fp32 below: two individually rounded operations per instruction)
        const uint64_t scale2 = pack_f32x2(scale_log2e, scale_log2e);
        const uint64_t neg_m2 = pack_f32x2(-m_ref, -m_ref);
        const uint64_t minus1 = pack_f32x2(-1.0f, -1.0f);
        uint64_t psum2 = pack_f32x2(0.0f, 0.0f);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t(&v)[32] = sv[h];
          uint32_t whi[16], wlo[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float a0, a1;
            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[2 * i]),
                                       __uint_as_float(v[2 * i + 1])),
                             scale2, neg_m2),
                a0, a1);
            const float p0 = ex2_approx(a0), p1 = ex2_approx(a1);
            const uint64_t p2 = pack_f32x2(p0, p1);
            psum2 = add_f32x2(psum2, p2);
            const uint32_t hi = cvt_bf16x2(p0, p1);
            // p - hi: one rounding, as the subtraction has
            float r0, r1;
            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(hi << 16),
                                       __uint_as_float(hi & 0xffff0000u)),
                             minus1, p2),
                r0, r1);
            whi[i] = hi;
            wlo[i] = cvt_bf16x2(r0, r1);
          }
          // P of 32 keys: hi in columns 0..15 of theirs, lo in 16..31 (the scores of those
          // columns are already consumed).
          tmem_st16(t_row + (uint32_t)(32 * h), whi);
          tmem_st16(t_row + (uint32_t)(32 * h) + 16u, wlo);
        }
        float ps0, ps1;
        unpack_f32x2(psum2, ps0, ps1);
        l_run = __fadd_rn(l_run, __fadd_rn(ps0, ps1));
        tmem_st_wait();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0)
          mbar_arrive(bar.p); // this warp's part of P is in tensor memory
      }
      ok = mbar_wait(bar.o, (n - 1u) & 1u, abortp, wait_ns) && ok; // the item's last P V
      tcgen05_fence_after();
      __syncwarp();
      uint32_t o[32];
      {
        uint32_t v[32];
        tmem_ld32(t_out, o); // P_hi V_hi + P_lo V_hi
        tmem_ld32(t_out + 64u, v); // P_hi V_lo
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float a, b;
          unpack_f32x2(add_f32x2(pack_f32x2(__uint_as_float(o[i]), __uint_as_float(o[i + 1])),
                           pack_f32x2(__uint_as_float(v[i]), __uint_as_float(v[i + 1]))),
              a, b);
          o[i] = __float_as_uint(a);
          o[i + 1] = __float_as_uint(b);
        }
      }
      tcgen05_fence_before(); // (what the next item's first arrival at bar.p publishes)

      // Row sum over both halves, then normalise.
      xch_sum[half][row] = l_run;
      pair_barrier(quad);
      const float inv = __fdiv_rn(1.0f, __fadd_rn(xch_sum[0][row], xch_sum[1][row]));
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float f = __fmul_rn(__uint_as_float(o[i]), inv);
        lo_run = fminf(lo_run, f);
        hi_run = fmaxf(hi_run, f);
        o[i] = __float_as_uint(f);
      }
      // The 128 x 64 result leaves through the K or the V buffers (att_loads): half 0's
      // 32 columns in the first 16 KiB tile, half 1's in the second, rows of 128 bytes in the
      // 128-byte swizzle pattern, one TMA store per tile, which writes whole lines.
      const bool in_v = nkb == 1;
      if (!in_v && item + gridDim.x < n_items)
        ok = mbar_wait(bar.s, n & 1u, abortp, wait_ns) && ok;
      const uint32_t my_row =
          (in_v ? (half ? tiles.vl : tiles.vh) : (half ? tiles.kl : tiles.kh)) + (uint32_t)row * 128u;
      const uint32_t swz = ((uint32_t)row & 7u) << 4;
#pragma unroll
      for (int i = 0; i < 32; i += 4)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(
                         my_row + (((uint32_t)i * 4u) ^ swz)),
                     "r"(o[i]), "r"(o[i + 1]), "r"(o[i + 2]), "r"(o[i + 3])
                     : "memory");
      fence_proxy_async_smem(); // the tiles were written through the generic proxy
      __syncwarp();
      if (lane == 0)
        mbar_arrive(bar.r);
    }
    if (__all_sync(0xffffffffu, ok) && out_range)
      range_commit_block(range, out_range, lo_run, hi_run, blockIdx.x);
  }

  // ---- teardown ----
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tcgen05_fence_after();
    tmem_dealloc(tmem, kTmemColsAtt);
  }
  if (tid == 0 && abort_flag)
    atomicExch(status, 1);
}

// x [rows, cols] fp32 with row pitch ld_x -> bf16 planes hi, lo [rows, ld_p]
// at column offset col0: hi = bf16(x), lo = bf16(x - hi).
__global__ void __launch_bounds__(256)
    split_bf16_kernel(const float *__restrict__ x, int64_t rows, int64_t cols,
        int64_t ld_x, __nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo,
        int64_t ld_p, int64_t col0) {
  const int64_t c4n = cols >> 2;
  const int64_t total = rows * c4n;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / c4n, c = (i % c4n) * 4;
    const float4 v = *reinterpret_cast<const float4 *>(x + r * ld_x + c);
    const uint32_t h0 = cvt_bf16x2(v.x, v.y), h1 = cvt_bf16x2(v.z, v.w);
    const uint32_t l0 = cvt_bf16x2(__fsub_rn(v.x, __uint_as_float(h0 << 16)),
        __fsub_rn(v.y, __uint_as_float(h0 & 0xffff0000u)));
    const uint32_t l1 = cvt_bf16x2(__fsub_rn(v.z, __uint_as_float(h1 << 16)),
        __fsub_rn(v.w, __uint_as_float(h1 & 0xffff0000u)));
    *reinterpret_cast<uint2 *>(hi + r * ld_p + col0 + c) = make_uint2(h0, h1);
    *reinterpret_cast<uint2 *>(lo + r * ld_p + col0 + c) = make_uint2(l0, l1);
  }
}

} // namespace

bool attention_tc_supported(int64_t B, int64_t S, int64_t heads, int64_t dh,
    int64_t ld_planes, int64_t ld_out, const void *hi, const void *lo,
    const float *out) {
  // OMCUDA_ATTENTION=mma|simt keeps the older kernels, to cross-check them.
  static const bool disabled = [] {
    const char *s = getenv("OMCUDA_ATTENTION");
    return s && (strcmp(s, "mma") == 0 || strcmp(s, "simt") == 0);
  }();
  if (disabled)
    return false;
  return dh == kTDh && S > 0 && S % kTK == 0 && B * heads > 0 &&
         B * S < (int64_t(1) << 31) && ld_planes % 8 == 0 && ld_out % 4 == 0 &&
         ((((uintptr_t)hi | (uintptr_t)lo | (uintptr_t)out) & 15u) == 0);
}

int launch_attention_tc(const void *hi, const void *lo, int64_t ld_planes,
    int64_t q_col, int64_t k_col, int64_t v_col, int64_t B, int64_t S,
    int64_t heads, float scale, float *out, int64_t ld_out, void *out_range,
    cudaStream_t st) {
  if ((q_col | k_col | v_col) % 8 != 0)
    return fail(OMCUDA_EINVAL, "Attention: column offsets must be multiples of 8");
  static PerDeviceInt attr_set;
  if (!attr_set.get()) {
    OMCUDA_CHECK(cudaFuncSetAttribute(attention_tc_kernel,
        cudaFuncAttributeMaxDynamicSharedMemorySize, kTcAttSmem));
    attr_set.set(1);
  }
  const int64_t T = B * S;
  CUtensorMap map_hi, map_lo, map_out;
  int rc = make_tma_map_2d(&map_hi, hi, T, ld_planes, ld_planes * 2, kTDh, kTK, 2, 128);
  if (rc != OMCUDA_OK)
    return rc;
  rc = make_tma_map_2d(&map_lo, lo, T, ld_planes, ld_planes * 2, kTDh, kTK, 2, 128);
  if (rc != OMCUDA_OK)
    return rc;
  // output: boxes of 128 rows x 32 fp32 columns (128-byte rows)
  rc = make_tma_map_2d(&map_out, out, T, heads * kTDh, ld_out * 4, 32, kTQ, 4, 128);
  if (rc != OMCUDA_OK)
    return rc;
  int *status = tc_status_word();
  if (!status)
    return fail(OMCUDA_ENOMEM, "Attention: cannot allocate the status word");
  const int64_t n_items = (S / kTQ) * B * heads;
  const float scale_log2e = scale * 1.4426950408889634f;
  // Persistent CTAs, two per SM, each walking its share of the
  // (batch, head, 128-query-row) items.
  const int64_t resident = (int64_t)sm_count() * 2;
  const unsigned grid = (unsigned)(n_items < resident ? n_items : resident);
  OMCUDA_CHECK(launch_pdl(attention_tc_kernel, grid, kTcAttThreads, kTcAttSmem, st, 0,
      pdl_pays(B * S * heads * kTDh), map_hi, map_lo, map_out, (int32_t)q_col,
      (int32_t)k_col, (int32_t)v_col, S, heads, n_items, scale_log2e,
      (uint32_t *)out_range, status, tc_wait_limit_ns()));
  OMCUDA_CHECK_LAUNCH("attention_tc_kernel");
  return OMCUDA_OK;
}

int launch_split_bf16(const float *x, int64_t rows, int64_t cols, int64_t ld_x,
    void *hi, void *lo, int64_t ld_p, int64_t col0, cudaStream_t st) {
  if (cols % 4 != 0 || ld_x % 4 != 0 || ld_p % 4 != 0 || col0 % 4 != 0 ||
      (((uintptr_t)x & 15u) != 0) || ((((uintptr_t)hi | (uintptr_t)lo) & 7u) != 0))
    return fail(OMCUDA_EINVAL, "SplitBf16: rows must be 16-byte aligned");
  const int64_t total = rows * (cols >> 2);
  if (total == 0)
    return OMCUDA_OK;
  int64_t want = ceil_div(total, 256 * 4);
  const int64_t cap = (int64_t)sm_count() * 8;
  split_bf16_kernel<<<(unsigned)(want < cap ? want : cap), 256, 0, st>>>(x, rows,
      cols, ld_x, (__nv_bfloat16 *)hi, (__nv_bfloat16 *)lo, ld_p, col0);
  OMCUDA_CHECK_LAUNCH("split_bf16_kernel");
  return OMCUDA_OK;
}

} // namespace omcuda

using namespace omcuda;

extern "C" int omcudaDevSplitBf16(const float *x, int64_t rows, int64_t cols,
    int64_t ld_x, void *hi, void *lo, int64_t ld_planes, int64_t col0,
    void *stream) {
  if (rows < 0 || cols < 0 || ld_x < cols || ld_planes < col0 + cols ||
      (rows > 0 && cols > 0 && (!x || !hi || !lo)))
    return fail(OMCUDA_EINVAL, "SplitBf16: bad argument");
  return launch_split_bf16(x, rows, cols, ld_x, hi, lo, ld_planes, col0,
      (cudaStream_t)stream);
}

extern "C" int omcudaDevAttentionBf16Supported(int64_t B, int64_t S,
    int64_t heads, int64_t dh, int64_t ld_planes, int64_t ld_out) {
  return attention_tc_supported(B, S, heads, dh, ld_planes, ld_out, nullptr,
             nullptr, nullptr)
             ? 1
             : 0;
}

extern "C" int omcudaDevAttentionBf16(const void *hi, const void *lo,
    int64_t ld_planes, int64_t q_col, int64_t k_col, int64_t v_col, int64_t B,
    int64_t S, int64_t heads, int64_t dh, float scale, float *out,
    int64_t ld_out, void *out_range, void *stream) {
  if (B < 0 || S <= 0 || heads <= 0 || !hi || !lo || !out || q_col < 0 ||
      k_col < 0 || v_col < 0 || ld_out < heads * dh ||
      ld_planes < heads * dh + (q_col > k_col ? (q_col > v_col ? q_col : v_col)
                                               : (k_col > v_col ? k_col : v_col)))
    return fail(OMCUDA_EINVAL, "AttentionBf16: bad argument");
  // The kernel takes the row maximum of the raw scores and scales it
  // afterwards, which equals the maximum of the scaled scores only for a
  // positive scale.
  if (!(scale > 0.0f) || !(scale < INFINITY))
    return fail(OMCUDA_EINVAL,
        "AttentionBf16: the scale must be positive and finite (got %g); "
        "omcudaDevAttention takes any scale", (double)scale);
  if (B == 0)
    return OMCUDA_OK;
  if (!attention_tc_supported(B, S, heads, dh, ld_planes, ld_out, hi, lo, out))
    return fail(OMCUDA_ENOTSUP,
        "AttentionBf16: needs head size 64, a sequence length that is a "
        "multiple of 128 and 16-byte aligned rows");
  return launch_attention_tc(hi, lo, ld_planes, q_col, k_col, v_col, B, S, heads,
      scale, out, ld_out, out_range, (cudaStream_t)stream);
}
