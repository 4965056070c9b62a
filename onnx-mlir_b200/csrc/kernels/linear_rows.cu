// Dynamic-quantized linear of up to 16 rows (decoding) in one launch:
// DynamicQuantizeLinear, MatMulInteger and the dequantize tail of
// gemm_epilogue.cuh, bit for bit what the kernels for each of them give.
//
// Bound by the read of the weight (K * N bytes of Bt, once).  As two kernels the
// weight waited for the whole activation to be quantized, in a launch whose few
// busy SMs had nothing to do with it.  Here a cluster of eight CTAs splits K: each
// asks for its slice of the weight columns it will need, reads its slice of x
// (every cluster all of it, so a byte of x is read once per cluster), the CTAs
// exchange their {min, max} through distributed shared memory, and each
// quantizes exactly the slice of x that its products need into its own shared
// memory: no scratch, and no quantized activation in global memory.  A warp then
// takes eight columns of a 64-column group at a time through
// mma.sync.m16n8k32 as gemm_i8_gemv_mma_kernel does (lane (g, q) loads 16 weight
// bytes of column g at offset 16 q of a 64-byte block of K, and A in the same
// order), and leaves its partial sums in shared memory.  When a cluster's columns
// are done, its CTAs share the outputs, each adding up the eight slices.
#include <cooperative_groups.h>

#include "../runtime/internal.h"
#include "gemm_epilogue.cuh"
#include "quantize.cuh"

namespace cg = cooperative_groups;

namespace omcuda {

namespace {

constexpr int kRowsMax = 16;
constexpr int kRowsCluster = 8;   // CTAs that split K
constexpr int kRowsThreads = 256; // eight warps, eight columns each
constexpr int kRowsGroup = 64;    // columns a CTA takes at a time
constexpr int kRowsUnroll = 8;    // 64-byte blocks of K in flight per warp
constexpr int kRowsHeld = 5;      // words of x a thread keeps: all of its slice
constexpr int kRowsMaxRounds = 8; // column groups per cluster
constexpr int64_t kRowsMaxSmem = 100 * 1024; // two CTAs per SM

// Bytes of K per CTA, and the pitch of its quantized rows: 16 banks apart modulo
// 32, so that two rows' 64-byte blocks take all of them.
__host__ __device__ inline int rows_slice(int64_t kp) {
  return (int)(ceil_div(kp, kRowsCluster * 64) * 64);
}
__host__ __device__ inline int rows_pitch(int slice) {
  return slice % 128 == 0 ? slice + 64 : slice;
}
int64_t rows_smem(int64_t kp, int rounds) {
  return (int64_t)kRowsMax * rows_pitch(rows_slice(kp)) +
         (int64_t)rounds * kRowsMax * kRowsGroup * 4;
}

} // namespace

template <bool kBSigned>
__global__ void __launch_bounds__(kRowsThreads, 2)
    linear_rows_kernel(const float *__restrict__ x, const uint8_t *__restrict__ Bt, int64_t kp,
        int vec_in, int rounds, int mode, EpiParams p) {
  extern __shared__ __align__(16) uint8_t rows_mem[];
  __shared__ float s_lo[kRowsThreads / 32], s_hi[kRowsThreads / 32];
  __shared__ float c_lo[kRowsCluster], c_hi[kRowsCluster];
  __shared__ int32_t s_rowsum[kRowsMax];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int64_t clusters = gridDim.x / kRowsCluster, first = blockIdx.x / kRowsCluster;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slice = rows_slice(kp), pitch = rows_pitch(slice);
  const int64_t k0 = (int64_t)rank * slice;
  const int len = (int)(kp - k0 < slice ? (kp > k0 ? kp - k0 : 0) : slice); // of Bt
  uint8_t *a_rows = rows_mem; // [16][pitch]
  int32_t *part = reinterpret_cast<int32_t *>(rows_mem + kRowsMax * pitch); // [rounds][16][64]
  // (the successor at the end, see GemmCall::early_next: 16 x 768 x 768 5.9 -> 5.7 us; not where
  // it may prefetch a weight meanwhile, 2 x 8192 x 8192 16.7 and 18.0)
  if (rounds > 1)
    pdl_sync();
  else
    pdl_wait();
  x = after_pdl(x);
  Bt = after_pdl(Bt);
  const EpiParams e = epi_after_pdl(p);
  // The warp's columns of round rd, 64-byte blocks b0 .. b0 + 7 of the slice, into
  // registers.  The first are asked for before x is looked at.  (Asking L2 for all of
  // them here, in pieces of a slice's size, made it slower: 1 x 4096 x 14336 20.0
  // against 15.1 us.)
  const int g = lane >> 2, q = lane & 3;
  uint4 bw[kRowsUnroll];
  const auto fetch = [&](int rd, int b0) {
    const int64_t n = (first + rd * clusters) * kRowsGroup + 8 * warp + g;
    // (columns past N re-read the last one)
    const uint8_t *brow = Bt + (n < p.N ? n : p.N - 1) * kp + k0 + 16 * q;
#pragma unroll
    for (int u = 0; u < kRowsUnroll; ++u)
      bw[u] = 64 * (b0 + u) + 16 * q < len
                  ? __ldcs(reinterpret_cast<const uint4 *>(brow + 64 * (b0 + u)))
                  : make_uint4(0, 0, 0, 0);
  };
  fetch(0, 0);
  cluster.barrier_arrive(); // "has started": waited for before the first remote store
  if (threadIdx.x < kRowsMax)
    s_rowsum[threadIdx.x] = 0;

  // ---- this CTA's slice of x: its range ----
  const int M = (int)p.M;
  const int words = len >> 2; // per row (len is a multiple of 16)
  const int total = M * words;
  const auto load = [&](int w) {
    const int r = w / words;
    const int64_t k = k0 + 4 * (w - r * words);
    const int64_t have = p.K - k;
    const float *src = x + r * p.K + k;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (have >= 4 && vec_in) {
      v = __ldg(reinterpret_cast<const float4 *>(src));
    } else {
      if (have > 0)
        v.x = __ldg(src);
      if (have > 1)
        v.y = __ldg(src + 1);
      if (have > 2)
        v.z = __ldg(src + 2);
      if (have > 3)
        v.w = __ldg(src + 3);
    }
    return v;
  };
  float lo = INFINITY, hi = -INFINITY;
  // (zeros that stand for no element change neither scalar: the range is widened
  // to hold 0 before anything is derived from it)
  const auto fold = [&](const float4 &v) {
    lo = min3f(min3f(lo, v.x, v.y), v.z, v.w);
    hi = max3f(max3f(hi, v.x, v.y), v.z, v.w);
  };
  float4 held[kRowsHeld];
#pragma unroll
  for (int u = 0; u < kRowsHeld; ++u) {
    const int w = threadIdx.x + u * kRowsThreads;
    held[u] = w < total ? load(w) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
#pragma unroll
  for (int u = 0; u < kRowsHeld; ++u)
    fold(held[u]);
  lo = warp_min(lo);
  hi = warp_max(hi);
  if (lane == 0) {
    s_lo[warp] = lo;
    s_hi[warp] = hi;
  }
  __syncthreads();
  cluster.barrier_wait();
  if (threadIdx.x < kRowsCluster) { // thread i tells CTA i
    lo = s_lo[0];
    hi = s_hi[0];
#pragma unroll
    for (int w = 1; w < kRowsThreads / 32; ++w) {
      lo = fminf(lo, s_lo[w]);
      hi = fmaxf(hi, s_hi[w]);
    }
    *cluster.map_shared_rank(&c_lo[rank], threadIdx.x) = lo;
    *cluster.map_shared_rank(&c_hi[rank], threadIdx.x) = hi;
  }
  cluster.sync();
  lo = c_lo[0];
  hi = c_hi[0];
#pragma unroll
  for (int i = 1; i < kRowsCluster; ++i) {
    lo = fminf(lo, c_lo[i]);
    hi = fmaxf(hi, c_hi[i]);
  }
  float scale, zp_f;
  dql_params_from_range(lo, hi, &scale, &zp_f, mode);
  const QuantConsts qc = make_quant_consts<false>(scale, zp_f, mode);

  // ---- quantized into shared memory ----
  const auto store = [&](int w, const float4 &v) {
    const int r = w / words, c = 4 * (w - r * words);
    const int64_t have = p.K - (k0 + c);
    uint32_t q = have > 0 ? quantize_four<false>(v, qc) : 0u;
    if (have > 0 && have < 4)
      q &= (1u << (8 * (int)have)) - 1u;
    *reinterpret_cast<uint32_t *>(a_rows + r * pitch + c) = q;
    if (e.b_zp_len != 0)
      atomicAdd(&s_rowsum[r], add_bytes<false>(q, 0));
  };
#pragma unroll
  for (int u = 0; u < kRowsHeld; ++u) {
    const int w = threadIdx.x + u * kRowsThreads;
    if (w < total)
      store(w, held[u]);
  }
  __syncthreads();

  // ---- products: rows 0..15 (those from M on are whatever the memory holds, and
  // never stored) times this CTA's slice of the cluster's columns ----
  const int blocks = (len + 63) >> 6;
  const uint8_t *arow = a_rows + g * pitch + 16 * q;
  for (int rd = 0; rd < rounds; ++rd) {
    if ((first + rd * clusters) * kRowsGroup >= p.N)
      break;
    int32_t acc[4] = {0, 0, 0, 0};
    for (int b0 = 0; b0 < blocks; b0 += kRowsUnroll) {
#pragma unroll
      for (int u = 0; u < kRowsUnroll; ++u) {
        if (b0 + u >= blocks)
          break;
        const uint4 a_lo = *reinterpret_cast<const uint4 *>(arow + 64 * (b0 + u));
        const uint4 a_hi = *reinterpret_cast<const uint4 *>(arow + 8 * pitch + 64 * (b0 + u));
        mma_m16n8k32<false, kBSigned>(acc, a_lo.x, a_hi.x, a_lo.y, a_hi.y, bw[u].x, bw[u].y);
        mma_m16n8k32<false, kBSigned>(acc, a_lo.z, a_hi.z, a_lo.w, a_hi.w, bw[u].z, bw[u].w);
      }
      if (b0 + kRowsUnroll < blocks)
        fetch(rd, b0 + kRowsUnroll);
      else if (rd + 1 < rounds)
        fetch(rd + 1, 0);
    }
    // c0,c1 = row g, columns 2q, 2q+1; c2,c3 = row g + 8
    int32_t *out = part + (rd * kRowsMax + g) * kRowsGroup + 8 * warp + 2 * q;
    *reinterpret_cast<int2 *>(out) = make_int2(acc[0], acc[1]);
    *reinterpret_cast<int2 *>(out + 8 * kRowsGroup) = make_int2(acc[2], acc[3]);
  }
  cluster.sync();

  // ---- outputs: this CTA's share of the cluster's, the eight slices added up ----
  EpiScalars sc;
  sc.sa = scale;
  sc.s0 = e.sb_len == 1 ? __fmul_rn(scale, __ldg(e.sb)) : 1.0f;
  sc.yz = 0;
  EpiRow row;
  row.az = (int32_t)zp_f;
  const int outs = rounds * M * kRowsGroup;
  for (int i = rank * kRowsThreads + (int)threadIdx.x; i < outs; i += kRowsCluster * kRowsThreads) {
    const int c = i % kRowsGroup, m = i / kRowsGroup % M, rd = i / kRowsGroup / M;
    const int64_t n = (first + rd * clusters) * kRowsGroup + c;
    if (n >= p.N)
      continue;
    int32_t sum = 0;
    row.rs = 0;
#pragma unroll
    for (int r = 0; r < kRowsCluster; ++r)
      sum += *cluster.map_shared_rank(part + (rd * kRowsMax + m) * kRowsGroup + c, r);
    if (e.b_zp_len != 0) {
#pragma unroll
      for (int r = 0; r < kRowsCluster; ++r)
        row.rs += *cluster.map_shared_rank(&s_rowsum[m], r);
    }
    uint32_t v = (uint32_t)sum - (uint32_t)row.az * (uint32_t)__ldg(e.colsum + n);
    if (e.b_zp_len != 0) {
      const uint32_t bz = (uint32_t)load_zp8(e.b_zp, e.b_zp_len == 1 ? 0 : n, e.b_signed);
      v += bz * ((uint32_t)p.K * (uint32_t)row.az - (uint32_t)row.rs);
    }
    reinterpret_cast<float *>(p.Y)[m * p.N + n] = epi_dequant(e, sc, (int32_t)v, n);
  }
  cluster.sync(); // nobody's sums may go before they have been read
}

namespace {

// Clusters of linear_rows_kernel that are resident at once.
int rows_clusters() {
  static PerDeviceInt cached;
  int n = cached.get();
  if (n == 0) {
    n = 1;
    cudaLaunchConfig_t q = {};
    q.gridDim = dim3((unsigned)(2 * sm_count() / kRowsCluster * kRowsCluster), 1, 1);
    q.blockDim = dim3(kRowsThreads, 1, 1);
    q.dynamicSmemBytes = kRowsMaxSmem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kRowsCluster;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    q.attrs = at;
    q.numAttrs = 1;
    int a = 0;
    if (cudaFuncSetAttribute(linear_rows_kernel<true>,
            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowsMaxSmem) == cudaSuccess &&
        cudaFuncSetAttribute(linear_rows_kernel<false>,
            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowsMaxSmem) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&a, linear_rows_kernel<true>, &q) == cudaSuccess && a > 0)
      n = a;
    (void)cudaGetLastError();
    cached.set(n);
  }
  return n;
}

int rows_rounds(int64_t N) {
  const int64_t groups = ceil_div(N, kRowsGroup), most = rows_clusters();
  return (int)ceil_div(groups, groups < most ? groups : most);
}

} // namespace

int linear_rows_groups(int64_t N) { return rows_rounds(N); }

bool linear_rows_wanted(int64_t M, int64_t N, int64_t kp) {
  // Every cluster reads all of x, so x has to be small next to the weight a cluster
  // reads: 16 x 256 x 256 5.8 us here and 7.0 as quantize and product, 16 x 768 x 768 5.8
  // and 7.5, 6 x 2062 x 1072 7.1 and 8.2.  One row is quantized so fast that the dp4a
  // kernel behind it is as good (1 x 2048 x 2048: 6.2 and 5.9).  The line was drawn
  // against the GEMV-shaped products, well inside: none of 710 sizes up to 32768 values
  // was more than 2 % faster as two kernels.  Against the few-rows kernel, which now makes
  // the product of large weights, that holds for one column group per cluster (0.55 to
  // 0.94 of the two kernels' time on 39 sizes), not for more (1.02 to 1.8 on 19): 2 x
  // 8192 x 8192 16.8 and 11.6 with the weight in L2, 19.5 and 16.7 beyond, 2 x 4096 x 14336
  // 15.4 and 11.0, 18.1 and 15.7, 15 x 2176 x 15360 17.4 and 9.7, 19.7 and 12.1, 5 x 1650 x 5419
  // 9.0 and 8.2, 9.3 and 8.2.  Calls with more that may take scratch are therefore two
  // kernels.  With zero points per column two would be faster as well (2 x 8192 x 8192 17.1 and 12.4,
  // 19.7 and 17.2), but such a call has always been one launch and is held to that by the test
  // that counts them (test_linear_of_few_rows_values).
  if (M < 2 || M > kRowsMax || N > (int64_t)1 << 24)
    return false;
  if (M * kp > 16384 && (M * kp > 32768 || N < 1024 * M))
    return false;
  // A thread holds its part of the slice: up to 1200 words a CTA within the line above
  // (15 x 2176), slices being rounded up to 64 values a row.
  if (M * (rows_slice(kp) / 4) > kRowsHeld * kRowsThreads)
    return false;
  // More than one column group per cluster: not for weights of a few MB (4 x 768 x 3072:
  // 7.1 us here, 6.9 as two kernels).
  const int rounds = rows_rounds(N);
  if (rounds > 1 && N * kp < (int64_t)8 << 20)
    return false;
  return rounds <= kRowsMaxRounds && rows_smem(kp, rounds) <= kRowsMaxSmem;
}

int launch_linear_rows(const float *x, const GemmCall &a, cudaStream_t st) {
  const int rounds = rows_rounds(a.N);
  const int64_t groups = ceil_div(a.N, kRowsGroup);
  const unsigned clusters = (unsigned)ceil_div(groups, rounds);
  const int vec_in = ((uintptr_t)x & 15u) == 0 && a.K % 4 == 0;
  OMCUDA_CHECK(launch_pdl(a.B.b_signed ? linear_rows_kernel<true> : linear_rows_kernel<false>,
      clusters * kRowsCluster, kRowsThreads, (size_t)rows_smem(a.B.kp, rounds), st, kRowsCluster,
      true, x, (const uint8_t *)a.B.bt, a.B.kp, vec_in, rounds, quant_mode(),
      make_epi_params(a)));
  count_launch();
  return OMCUDA_OK;
}

} // namespace omcuda
