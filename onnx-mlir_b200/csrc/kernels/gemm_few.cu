// int8 x int8 -> int32 GEMM of few rows of A (decoding, short requests) on the
// tensor cores: the semantics and tails of gemm_tc.cu, bit for bit.
//
// Bound by the read of the weight (K * N bytes of Bt, once), which a few rows do
// not amortise, and at small sizes by latency: of launches, and of what has to happen in
// turn inside one.  So the operands change places: a tile is 128 output columns (rows of
// Bt, the MMA's M) by T rows of A (its N, 16 to 128), which wastes little on rows that do
// not exist, and the K loop of a tile is dealt to the CTAs of a cluster, so that more SMs
// read: as many as few_plan() finds cheapest, which for clusters of three and more counts on
// three quarters of the SMs (16 x 14336 x 4096: 32 tiles, 96 CTAs in clusters of three).  A CTA
// lives for one slice of one tile, several are resident per SM:
//   warp 8      asks for the slices of Bt as soon as it starts, before the kernel it
//               follows has finished (see `settled`), and for A behind pdl_sync()
//   warp 9      issues the MMAs, four K slices of 32 bytes per block of 128, two blocks
//               per stage: what its thread spends on a stage besides (a wait, a commit)
//               is as long as the four MMAs of a block (one block per stage: 0.34 us a
//               block, two 0.23; 16 x 14336 x 4096 on 64 CTAs 24.7 -> 21.5 us, 128 x 14336 x
//               4096 29.8 -> 27.3)
//   warps 0-7   read the sums out of tensor memory and send each row's to the CTA of
//               the cluster that owns the row; the owners add up what came and run
//               the tail, whole lines of Y at a time
// Sums of integers are exact in any order.
//
// Every wait on an mbarrier is bounded as in gemm_tc.cu; cluster barriers are
// reached by every thread whatever happens.
#include <cuda.h>

#include "../runtime/internal.h"
#include "gemm_epilogue.cuh"
#include "tc_ptx.cuh"

namespace omcuda {

namespace {

constexpr int kFewCols = 128;                 // output columns per tile
constexpr int kFewBK = 128;                   // bytes of K per block, a row of a swizzled tile
constexpr int kFewWBytes = kFewCols * kFewBK; // of Bt per block
constexpr int kFewBlocks = 2;                 // K blocks per stage
constexpr int kFewMaxStages = 6;
constexpr int64_t kFewMaxRows = 640;
constexpr int kFewWarps = 8; // that run the tail
constexpr int kFewThreads = 32 * (kFewWarps + 2);

// Publishes no memory of the thread, only that it has come this far, so it does not ask
// for release: that waits for all that the thread has in flight, one to three us here.
// (mbarriers: fence.mbarrier_init; the sums: the mbarrier that counts their bytes.)
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
                 "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}

__device__ __forceinline__ uint4 ld_shared_u4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ void st_shared_u32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Shared memory of this CTA to a CTA of the cluster; the bytes are counted on an
// mbarrier over there.  Both addresses and the size are multiples of 16.
__device__ __forceinline__ void copy_to_cluster(
    uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes"
      " [%0], [%1], %2, [%3];" ::"r"(dst),
      "r"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// What four neighbouring output columns need, held by the thread that makes them.
struct FewColumns {
  uint32_t colsum[4], bz[4];
  float scale[4]; // form 0 and REQUANT: the factor; form 1: the second one
  float bias[4];
};

// Columns past N work on the last one and are not stored.
template <int EPI>
__device__ __forceinline__ FewColumns few_columns(
    const EpiParams &p, const EpiScalars &sc, int64_t n0) {
  FewColumns c;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int64_t n = n0 + j < p.N ? n0 + j : p.N - 1;
    c.colsum[j] = p.a_zp_len != 0 ? (uint32_t)__ldg(p.colsum + n) : 0u;
    c.bz[j] = p.b_zp_len != 0
                  ? (uint32_t)load_zp8(p.b_zp, p.b_zp_len == 1 ? 0 : n, p.b_signed)
                  : 0u;
    c.scale[j] = EPI == OMCUDA_EPI_I32 ? 1.0f : __ldg(p.sb + (p.sb_len == 1 ? 0 : n));
    c.bias[j] = epi_is_dequant(EPI) && p.bias ? __ldg(p.bias + n) : 0.0f;
    if (epi_is_dequant(EPI) && p.form == 0) // onnx.Mul of the two scales
      c.scale[j] = __fmul_rn(sc.sa, c.scale[j]);
  }
  return c;
}

// Behind a wait that gave up: until the copies that `bar` counts have landed, or the
// limit is over once more, so that none of them writes to memory the CTA has left.
__device__ __forceinline__ void few_drain(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
  const uint64_t start = global_timer();
  while (!mbar_try_wait(bar, parity) && global_timer() - start <= limit_ns) {
  }
}

// Four outputs of a row: epi_int and the tails of gemm_epilogue.cuh on values that are
// held.  valid: columns that exist; whole: all four, in a Y that takes them together.
template <int EPI>
__device__ __forceinline__ void few_outputs(const EpiParams &p, const EpiScalars &sc,
    const FewColumns &c, const EpiRow &row, uint4 acc, int64_t at, int valid, bool whole,
    float &lo, float &hi) {
  uint32_t v[4] = {acc.x, acc.y, acc.z, acc.w};
  // (products with zero points that are absent are products with zero)
  const uint32_t tr = (uint32_t)p.K * (uint32_t)row.az - (uint32_t)row.rs;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    v[j] = v[j] - (uint32_t)row.az * c.colsum[j] + c.bz[j] * tr;
  if (EPI == OMCUDA_EPI_I32) {
    uint32_t *dst = reinterpret_cast<uint32_t *>(p.Y) + at;
    if (whole)
      *reinterpret_cast<uint4 *>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
    else
      for (int j = 0; j < valid; ++j)
        dst[j] = v[j];
    return;
  }
  if (EPI == OMCUDA_EPI_REQUANT) {
    uint32_t w = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float r = round_even(__fmul_rn(__int2float_rn((int32_t)v[j]), c.scale[j]));
      w |= (((uint32_t)__float2int_rz(r) + sc.yz) & 0xffu) << (8 * j);
    }
    uint8_t *dst = reinterpret_cast<uint8_t *>(p.Y) + at;
    if (whole)
      *reinterpret_cast<uint32_t *>(dst) = w;
    else
      for (int j = 0; j < valid; ++j)
        dst[j] = (uint8_t)(w >> (8 * j));
    return;
  }
  float y[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float f = __int2float_rn((int32_t)v[j]);
    y[j] = p.form == 0 ? __fmul_rn(f, c.scale[j]) : __fmul_rn(__fmul_rn(f, sc.sa), c.scale[j]);
  }
  if (p.bias) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      y[j] = __fadd_rn(y[j], c.bias[j]);
  }
  if (p.gelu) {
    gelu_erf_x2(y[0], y[1]);
    gelu_erf_x2(y[2], y[3]);
  }
  if (EPI == OMCUDA_EPI_DEQUANT_SPLIT) {
    // hi = bf16(y), lo = bf16(y - hi)
    uint32_t h[2], l[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h[j]) : "f"(y[2 * j + 1]), "f"(y[2 * j]));
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;"
          : "=r"(l[j])
          : "f"(__fsub_rn(y[2 * j + 1], __uint_as_float(h[j] & 0xffff0000u))),
          "f"(__fsub_rn(y[2 * j], __uint_as_float(h[j] << 16))));
    }
    uint16_t *dhi = reinterpret_cast<uint16_t *>(p.Y) + at, *dlo = dhi + p.M * p.N;
    if (whole) {
      *reinterpret_cast<uint2 *>(dhi) = make_uint2(h[0], h[1]);
      *reinterpret_cast<uint2 *>(dlo) = make_uint2(l[0], l[1]);
    } else {
      for (int j = 0; j < valid; ++j) {
        dhi[j] = (uint16_t)(h[j >> 1] >> (16 * (j & 1)));
        dlo[j] = (uint16_t)(l[j >> 1] >> (16 * (j & 1)));
      }
    }
  } else {
    float *dst = reinterpret_cast<float *>(p.Y) + at;
    if (p.residual) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < valid)
          y[j] = __fadd_rn(y[j], __ldg(p.residual + at + j));
    }
    if (whole)
      *reinterpret_cast<float4 *>(dst) = make_float4(y[0], y[1], y[2], y[3]);
    else
      for (int j = 0; j < valid; ++j)
        dst[j] = y[j];
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j < valid) {
      lo = fminf(lo, y[j]);
      hi = fmaxf(hi, y[j]);
    }
}

} // namespace

// grid: (tiles of N) * split by tiles of M; a cluster is the `split` CTAs of a tile.
// settled: Bt is not written by a kernel that may still be running when this one is set
// up, so it may be read before pdl_sync().
template <int T, int EPI>
__global__ void __launch_bounds__(kFewThreads, 3)
    gemm_i8_few_kernel(const __grid_constant__ CUtensorMap map_w,
        const __grid_constant__ CUtensorMap map_x, EpiParams p, uint32_t idesc,
        int split, int stages, int ring_bytes, int settled, int *status, uint64_t wait_ns) {
  constexpr int kXBytes = T * kFewBK;
  constexpr int kBlockBytes = kFewWBytes + kXBytes;
  constexpr int kStageBytes = kFewBlocks * kBlockBytes;
  constexpr int kTmemCols = T < 32 ? 32 : T;
  constexpr int kShare = T / 2; // rows a warp reads out of tensor memory

  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[kFewMaxStages];
  __shared__ uint64_t bar_empty[kFewMaxStages];
  __shared__ uint64_t bar_done; // all MMAs
  __shared__ uint64_t bar_sums; // what the cluster sends has come
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ RangeBlock range;

  const int tid = threadIdx.x, warp = warp_number(), lane = tid & 31;
  const int rank = split > 1 ? (int)cluster_ctarank() : 0;
  const int64_t n0 = (int64_t)(blockIdx.x / (unsigned)split) * kFewCols;
  const int64_t m0 = (int64_t)blockIdx.y * T;
  const int num_kb = (int)ceil_div(p.K, kFewBK);
  const int kb0 = (int)((int64_t)rank * num_kb / split);
  const int kbs = (int)((int64_t)(rank + 1) * num_kb / split) - kb0;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int64_t left = p.M - m0;
  const int rows = (int)(left < T ? left : T);
  const int own = (rows + split - 1) / split; // rows per CTA of the cluster
  const int first = rank * own;
  const int count = rows - first < own ? (rows > first ? rows - first : 0) : own;
  // This CTA's sums, [rows][128], take the place of the stages; behind those lies what
  // comes from the cluster, [split][count][128].
  const uint32_t mine = smem_base;
  const uint32_t sums = split > 1 ? smem_base + (uint32_t)ring_bytes : mine;
  volatile int *abortp = &abort_flag;
  const int steps = (kbs + kFewBlocks - 1) / kFewBlocks; // (the last may be one block short)
  const int ahead = steps < stages ? steps : stages;
  // Step i's loads, the weight's or the activations', into stage s.
  const auto load_w = [&](int i, int s) {
    for (int b = 0; b < kFewBlocks && kFewBlocks * i + b < kbs; ++b)
      tma_load_2d(smem_base + s * kStageBytes + b * kBlockBytes, &map_w,
          (kb0 + kFewBlocks * i + b) * kFewBK, (int32_t)n0, smem_u32(&bar_full[s]));
  };
  const auto load_x = [&](int i, int s) {
    for (int b = 0; b < kFewBlocks && kFewBlocks * i + b < kbs; ++b)
      tma_load_2d(smem_base + s * kStageBytes + b * kBlockBytes + kFewWBytes, &map_x,
          (kb0 + kFewBlocks * i + b) * kFewBK, (int32_t)m0, smem_u32(&bar_full[s]));
  };
  const auto expect = [&](int i, int s) {
    const int blocks = kbs - kFewBlocks * i < kFewBlocks ? kbs - kFewBlocks * i : kFewBlocks;
    mbar_expect_tx(smem_u32(&bar_full[s]), (uint32_t)(blocks * kBlockBytes));
  };

  if (warp == kFewWarps && elect_one()) {
    abort_flag = 0;
    range_block_init(range, kFewWarps);
    for (int s = 0; s < ahead; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    mbar_init(smem_u32(&bar_done), 1);
    mbar_init(smem_u32(&bar_sums), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (split > 1)
      mbar_expect_tx(smem_u32(&bar_sums), (uint32_t)(split * count * kFewCols * 4));
    // (the stages only: the rest of the slice asked for in L2 as well, by TMA or by the idle
    // warps' prefetch instructions, 16 x 14336 x 4096 19.4 -> 21.4 us)
    if (settled)
      for (int s = 0; s < ahead; ++s) {
        expect(s, s);
        load_w(s, s);
      }
    prefetch_tensormap(&map_x);
  }
  if (warp == kFewWarps + 1)
    tmem_alloc(smem_u32(&tmem_base_slot), kTmemCols);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  if (split > 1)
    cluster_arrive(); // "has started": waited for before the first copy
  if (p.early_next)
    pdl_sync();
  else
    pdl_wait();
  const EpiParams e = epi_after_pdl(p);

  if (warp == kFewWarps) {
    // ---------------- loads ----------------
    if (elect_one()) {
      for (int s = 0; s < ahead; ++s) {
        if (!settled) {
          expect(s, s);
          load_w(s, s);
        }
        load_x(s, s);
      }
      int stage = 0, asked = ahead; // (stage: of the next load)
      uint32_t phase = 0;
      for (int i = ahead; i < steps; ++i, ++asked) {
        if (!mbar_wait(smem_u32(&bar_empty[stage]), phase, abortp, wait_ns))
          break;
        expect(i, stage);
        load_w(i, stage);
        load_x(i, stage);
        if (++stage == ahead) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (!mbar_wait(smem_u32(&bar_done), 0, abortp, wait_ns))
        for (int i = asked - ahead; i < asked; ++i)
          few_drain(smem_u32(&bar_full[i % ahead]), (uint32_t)(i / ahead) & 1u, wait_ns);
    }
  } else if (warp == kFewWarps + 1) {
    // ---------------- MMAs ----------------
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true, landed = false; // (asked one stage ahead, as in gemm_tc.cu)
      for (int i = 0; i < steps; ++i) {
        ok = landed || mbar_wait(smem_u32(&bar_full[stage]), phase, abortp, wait_ns);
        if (!ok)
          break;
        const int nstage = stage + 1 == ahead ? 0 : stage + 1;
        const uint32_t nphase = nstage == 0 ? phase ^ 1u : phase;
        landed = mbar_test_wait(smem_u32(&bar_full[nstage]), nphase);
        tcgen05_fence_after();
        const uint32_t sw = smem_base + stage * kStageBytes;
        static_assert(kFewBK == 128, "four K slices per block");
        umma_i8_x4(tmem_base, make_smem_desc(sw), make_smem_desc(sw + kFewWBytes), idesc,
            i != 0 ? 1u : 0u);
        if (kFewBlocks * i + 1 < kbs)
          umma_i8_x4(tmem_base, make_smem_desc(sw + kBlockBytes),
              make_smem_desc(sw + kBlockBytes + kFewWBytes), idesc, 1u);
        if (i + ahead < steps)
          umma_commit(smem_u32(&bar_empty[stage]));
        stage = nstage;
        phase = nphase;
      }
      if (ok)
        umma_commit(smem_u32(&bar_done));
    }
  }

  const EpiScalars sc = epi_scalars(e);
  const EpiRow row0 = epi_row(e, m0); // (alike for all rows unless something is per row)
  const bool per_row = p.a_zp_len > 1 || p.b_zp_len != 0;
  const int64_t n = n0 + 4 * lane;
  const FewColumns col = few_columns<EPI>(e, sc, n);
  __syncwarp();

  // ---------------- tail ----------------
  float lo = INFINITY, hi = -INFINITY;
  bool ok = mbar_wait(smem_u32(&bar_done), 0, abortp, wait_ns);
  tcgen05_fence_after();
  if (ok && warp < kFewWarps) {
    const int quad = warp & 3; // TMEM lanes a warp may read
    const int r_lo = (warp >> 2) * kShare;
    constexpr int kRead = kShare < 32 ? 8 : 32;
    for (int r0 = r_lo; r0 < r_lo + kShare && r0 < rows; r0 += kRead) {
      uint32_t v[kRead];
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)r0;
      if constexpr (kRead == 8)
        tmem_ld8(taddr, v);
      else
        tmem_ld32(taddr, v);
      tmem_ld_wait();
      const uint32_t dst = mine + 4u * (uint32_t)(r0 * kFewCols + quad * 32 + lane);
#pragma unroll
      for (int j = 0; j < kRead; ++j)
        st_shared_u32(dst + 4u * kFewCols * j, v[j]);
    }
  }
  if (split > 1) {
    fence_proxy_async_smem(); // the sums were written through the generic proxy
    cluster_wait();           // every CTA of the cluster has started
    __syncthreads();
    if (tid < split && ok) { // thread i sends CTA i its rows
      const int from = tid * own, len = rows - from < own ? rows - from : own;
      if (len > 0)
        copy_to_cluster(mapa_shared(sums + 4u * (uint32_t)(rank * len * kFewCols), (uint32_t)tid),
            mine + 4u * (uint32_t)(from * kFewCols), (uint32_t)(len * kFewCols * 4),
            mapa_shared(smem_u32(&bar_sums), (uint32_t)tid));
    }
    if (!mbar_wait(smem_u32(&bar_sums), 0, abortp, wait_ns)) {
      ok = false;
      if (tid == 0) // (nor may the senders go while their copies come in here)
        few_drain(smem_u32(&bar_sums), 0, wait_ns);
    }
    cluster_arrive(); // "has its sums": waited for before this CTA's may go
  } else {
    __syncthreads();
  }
  const int valid = (int)(p.N - n < 4 ? p.N - n : 4);
  if (ok && valid > 0 && warp < kFewWarps) {
    const int esize = EPI == OMCUDA_EPI_REQUANT ? 1 : EPI == OMCUDA_EPI_DEQUANT_SPLIT ? 2 : 4;
    const bool whole = valid == 4 && (p.N & 3) == 0 &&
                       ((uintptr_t)p.Y & (uintptr_t)(4 * esize - 1)) == 0 &&
                       (EPI != OMCUDA_EPI_DEQUANT_SPLIT || ((p.M * p.N) & 3) == 0);
    const uint32_t from = sums + 16u * (uint32_t)lane;
    for (int i = warp; i < count; i += kFewWarps) {
      uint4 v = ld_shared_u4(from + 4u * (uint32_t)(i * kFewCols));
      for (int s = 1; s < split; ++s) {
        const uint4 w = ld_shared_u4(from + 4u * (uint32_t)((s * count + i) * kFewCols));
        v.x += w.x;
        v.y += w.y;
        v.z += w.z;
        v.w += w.w;
      }
      const int64_t m = m0 + first + i;
      const EpiRow row = per_row ? epi_row(e, m) : row0;
      few_outputs<EPI>(e, sc, col, row, v, m * p.N + n, valid, whole, lo, hi);
    }
  }
  if (epi_is_dequant(EPI) && p.out_range && warp < kFewWarps)
    range_commit_block(range, p.out_range, lo, hi, blockIdx.y * gridDim.x + blockIdx.x);

  // ---------------- teardown ----------------
  if (split > 1)
    cluster_wait();
  tcgen05_fence_before();
  __syncthreads();
  if (warp == kFewWarps + 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  if (tid == 0 && abort_flag)
    atomicExch(status, 1);
}

namespace {

// Instruction descriptor of tcgen05.mma kind::i8: s32 accumulator, M = 128 rows of Bt
// by t rows of A, both K-major.
uint32_t few_idesc(int w_signed, int x_signed, int t) {
  return 2u << 4 | (w_signed ? 1u : 0u) << 7 | (x_signed ? 1u : 0u) << 10 |
         (uint32_t)(t >> 3) << 17 | (uint32_t)(kFewCols >> 4) << 24;
}

struct FewPlan {
  int t, split, stages;
};

constexpr int64_t kFewSmemPerSm = 228 * 1024, kFewMaxSmem = 226 * 1024;

// Bytes of the stages, which the sums of the tile take the place of, and what the CTA
// needs besides.
int64_t few_ring(int t, int64_t stages) {
  const int64_t ring = stages * kFewBlocks * (kFewWBytes + t * kFewBK), tile = (int64_t)t * kFewCols * 4;
  return ring > tile ? ring : tile;
}
int64_t few_besides(int t, int split) {
  return 1024 + (split > 1 ? (int64_t)split * ((t + split - 1) / split) * kFewCols * 4 : 0);
}

template <int T, int EPI>
int launch_few_t(const GemmCall &a, const FewPlan &plan, cudaStream_t st) {
  static PerDeviceInt attr_set;
  if (!attr_set.get()) {
    OMCUDA_CHECK(cudaFuncSetAttribute(gemm_i8_few_kernel<T, EPI>,
        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFewMaxSmem));
    attr_set.set(1);
  }
  CUtensorMap map_w, map_x;
  int rc = make_tma_map_2d(&map_w, a.B.bt, a.N, a.B.kp, a.B.kp, kFewBK, kFewCols, 1, 128);
  if (rc == OMCUDA_OK)
    rc = make_tma_map_2d(&map_x, a.A, a.M, a.K, a.lda, kFewBK, T, 1, 128);
  if (rc != OMCUDA_OK)
    return rc;
  int *status = tc_status_word();
  if (!status)
    return fail(OMCUDA_ENOMEM, "GemmI8: cannot allocate the status word");
  const int64_t ring = few_ring(T, plan.stages);
  OMCUDA_CHECK(launch_pdl(gemm_i8_few_kernel<T, EPI>,
      dim3((unsigned)(ceil_div(a.N, kFewCols) * plan.split), (unsigned)ceil_div(a.M, T), 1),
      kFewThreads, (size_t)(ring + few_besides(T, plan.split)), st,
      plan.split > 1 ? plan.split : 0, true, map_w, map_x, make_epi_params(a),
      few_idesc(a.B.b_signed, a.a_signed, T), plan.split, plan.stages, (int)ring,
      a.b_settled ? 1 : 0, status, tc_wait_limit_ns()));
  count_launch();
  return OMCUDA_OK;
}

template <int EPI>
int launch_few_epi(const GemmCall &a, const FewPlan &plan, cudaStream_t st) {
  switch (plan.t) {
  case 16:
    return launch_few_t<16, EPI>(a, plan, st);
  case 32:
    return launch_few_t<32, EPI>(a, plan, st);
  case 64:
    return launch_few_t<64, EPI>(a, plan, st);
  default:
    return launch_few_t<128, EPI>(a, plan, st);
  }
}

// How the rows are cut into tiles of t and the K loop into `split`, by what a launch of
// such CTAs takes in us, fitted to 10000 launches (M 1 to 512, K and N 256 to 14336, all t
// and split, weights in L2 or not): the choice takes 1.1 % more than the best one in the
// mean, 18 % at most.
// The search runs on the host in every call: 32-bit divisions, and none where one round of
// CTAs does (128 x 768 x 768, 24 cuts: 0.54 -> 0.18 us of a 2.7 GHz core).
FewPlan few_plan(int64_t M, int64_t N, int64_t K) {
  const uint32_t num_kb = (uint32_t)ceil_div(K, kFewBK);
  const int64_t col_tiles = ceil_div(N, kFewCols);
  const int sm = sm_count();
  const auto ceil_few = [](int64_t a, int64_t b) { return a <= b ? 1 : ceil_div(a, b); };
  FewPlan best = {0, 0, 0};
  double least = 0.0;
  for (int t = 16; t <= 128 && (t == 16 || t < 2 * M); t *= 2) {
    const int64_t tiles = col_tiles * ((uint32_t)(M + t - 1) / (uint32_t)t);
    for (int split : {1, 2, 3, 4, 6, 8}) {
      if ((uint32_t)split > num_kb)
        break;
      const int64_t ctas = tiles * split;
      const int kbs = (int)((num_kb + split - 1) / (uint32_t)split);
      // SMs that clusters find together: with one CTA to an SM 16 clusters of eight, 32 of
      // four or 46 of three do not always fit, and the launch takes two rounds (64 x
      // 1536 x 6144 in 48 clusters of three 17.5 us, of two 12.2).
      const int64_t sms = sm * (split > 2 ? 3 : 4) / 4 - (split == 2 ? 8 : 0);
      // Stages: as many as the slice has, while all CTAs that an SM gets (three at most:
      // registers) fit.
      const int64_t wanted = ctas <= sms ? 1 : ctas <= 2 * sms ? 2 : 3;
      const int steps = (kbs + kFewBlocks - 1) / kFewBlocks;
      int stages = steps < kFewMaxStages ? steps : kFewMaxStages;
      const int64_t besides = few_besides(t, split) + 1024;
      int64_t smem;
      for (;; --stages) {
        smem = few_ring(t, stages) + besides;
        if (stages <= 1 || (smem <= kFewMaxSmem && smem * wanted <= kFewSmemPerSm))
          break;
      }
      if (smem > kFewMaxSmem)
        continue;
      const int64_t fit = 3 * smem <= kFewSmemPerSm ? 3 : 2 * smem <= kFewSmemPerSm ? 2 : 1;
      const int64_t rounds = ceil_few(ctas, sms * fit);
      const double per_sm = (double)ceil_few(rounds == 1 ? ctas : ceil_div(ctas, rounds), sm);
      const double load = per_sm * kbs * (16.0 + t / 8.0) * 0.0014; // KiB
      const double mma = per_sm * kbs * 0.07;
      const double chain = steps * 0.109 * (1.0 + 3.86 / stages);
      const double tail = per_sm * (t < M ? t : M) * 0.0229;
      const double us = rounds * ((load > mma ? (load > chain ? load : chain)
                                              : (mma > chain ? mma : chain)) + tail) +
                        ctas * 0.0037;
      if (best.t == 0 || us < least) {
        best = FewPlan{t, split, stages};
        least = us;
      }
    }
  }
  return best;
}

} // namespace

// Lines from 650 drawn linears and 320 of a grid (weights i8 and u8, in L2 or not; us of
// the call with the kernels that had it before and with this one, weights in L2).
bool gemm_few_wanted(int64_t M, int64_t N, int64_t K) {
  if (M > kFewMaxRows)
    return false;
  // Against the 128- and 256-row tiles of gemm_tc.cu: 32 x 8192 x 1127 28.3 -> 10.6, 61 x
  // 3072 x 768 15.5 -> 9.7, 103 x 1664 x 1997 14.0 -> 11.5, 64 x 512 x 512 9.0 -> 7.6.  Outputs that the
  // products do not make up for are better off in their tail: 345 x 281 x 3968 11 and 16, 94 x
  // 768 x 7424 12.0 and 13.3.  Nor is it for many rows of a large weight, which every tile of
  // rows reads again (79 x 4215 x 7488 20.2 and 21.8, 133 x 8386 x 5312 32.8 and 35.9).
  if (M > 16)
    return M <= 64 || (M * N <= 300000 + 200 * K && K * N <= 30000000);
  // Against the kernels for 2 to 16 rows, which have less to set up: worth it where there
  // is much to add up, or more columns than they find blocks for.  15 x 11584 x 360 16.3 ->
  // 10.6, 4 x 11456 x 1006 14.2 -> 9.1, 7 x 320 x 10597 11.8 -> 6.7, 10 x 3072 x 864 9.0 -> 7.8, but
  // 10 x 320 x 4480 7.2 and 7.9, 16 x 768 x 3776 7.5 and 7.7.  One row is read as fast without
  // tensor cores (1 x 4096 x 14336 17.3 and 17.6).
  return M > 1 && (N >= 4800 || K >= 2304);
}

void gemm_few_plan(int64_t M, int64_t N, int64_t K, int *rows, int *split) {
  const FewPlan plan = few_plan(M, N, K);
  *rows = plan.t;
  *split = plan.split;
}

bool gemm_few_supported(const GemmCall &a) {
  return (a.epilogue == OMCUDA_EPI_I32 || a.epilogue == OMCUDA_EPI_DEQUANT ||
             a.epilogue == OMCUDA_EPI_REQUANT || a.epilogue == OMCUDA_EPI_DEQUANT_SPLIT) &&
         a.M <= kFewMaxRows && gemm_tc_supported(a);
}

int launch_gemm_few(const GemmCall &a, cudaStream_t st) {
  const FewPlan plan = few_plan(a.M, a.N, a.K);
  switch (a.epilogue) {
  case OMCUDA_EPI_I32:
    return launch_few_epi<OMCUDA_EPI_I32>(a, plan, st);
  case OMCUDA_EPI_DEQUANT:
    return launch_few_epi<OMCUDA_EPI_DEQUANT>(a, plan, st);
  case OMCUDA_EPI_REQUANT:
    return launch_few_epi<OMCUDA_EPI_REQUANT>(a, plan, st);
  case OMCUDA_EPI_DEQUANT_SPLIT:
    return launch_few_epi<OMCUDA_EPI_DEQUANT_SPLIT>(a, plan, st);
  default:
    return fail(OMCUDA_EINVAL, "GemmI8: unknown epilogue %d", a.epilogue);
  }
}

} // namespace omcuda
