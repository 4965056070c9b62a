// Internal host-side interfaces shared by libomcuda's translation units.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "omcuda.h"

namespace omcuda {

int ensure_init();
bool sticky_error();
cudaStream_t current_stream();
// Device-memory pool with stream-ordered reuse.  The plain forms use the
// calling thread's stream (omcudaGetStream); the _on forms name the stream the
// block will be / was last used on.  optional: lack of memory is not recorded as an error.
void *pool_alloc(size_t bytes);
void pool_free(void *p);
void *pool_alloc_on(size_t bytes, cudaStream_t st, bool optional = false);
void pool_free_on(void *p, cudaStream_t st);
bool pool_owns(const void *p);

// Index of the device current on the calling thread, or -1.
constexpr int kMaxDevices = 64;
int current_device_index();
// A value a kernel's launcher computes once per device (launch attributes
// set, cluster occupancy); 0 means "not yet".  Safe to use from several host
// threads and with several devices in one process.
struct PerDeviceInt {
  int v[kMaxDevices] = {0};
  int get();
  void set(int x);
};

// OMCUDA_MODE_* flags set with omcudaSetQuantizationMode (process wide).
int quant_mode();

// Wait limit the tensor-core kernels are launched with (gemm_tc.cu).
uint64_t tc_wait_limit_ns();

// Whether two ranges of memory share a byte.
inline bool ranges_overlap(const void *a, int64_t a_bytes, const void *b, int64_t b_bytes) {
  const uintptr_t p = (uintptr_t)a, q = (uintptr_t)b;
  return a_bytes > 0 && b_bytes > 0 && p < q + (uintptr_t)b_bytes &&
         q < p + (uintptr_t)a_bytes;
}

// dql.cu
//
// DynamicQuantizeLinear of a [rows, cols] matrix into rows of `pitch` bytes (a
// multiple of 16, y 16-byte aligned), the tail of a row zero: the form the GEMM
// kernels take.  rowsum (i32 [rows], sums of a row's bytes) may be null; scratch
// as for omcudaDevDynamicQuantizeLinear.
int launch_dql_rows(const float *x, int64_t rows, int64_t cols, int64_t pitch, uint8_t *y,
    int32_t *rowsum, float *y_scale, uint8_t *y_zp, void *scratch, cudaStream_t st);

// omcudaDevDynamicQuantizeLinear; alone: as an operator by itself.
int launch_dql(const float *x, int64_t n, uint8_t *y, float *y_scale, uint8_t *y_zp,
    void *scratch, cudaStream_t st, bool alone);

// The same in one launch, without scratch, for a tensor that one cluster holds in
// its registers.  [rows, cols] into rows of `pitch` bytes as above, or one row
// of pitch == cols of any alignment.
bool dql_small_wanted(int64_t rows, int64_t pitch);
int launch_dql_small(const float *x, int64_t rows, int64_t cols, int64_t pitch,
    uint8_t *y, int32_t *rowsum, float *y_scale, uint8_t *y_zp, cudaStream_t st);
// Whether launch_dql_small takes a flat tensor of n values at all.  Up to four times
// the size that is faster so, it serves calls for which the two passes are wrong:
// one on a stream that is being captured, whose replays would write the partials to
// a pool block that was given back, and one that writes onto x, which the second
// pass reads again.
bool dql_one_cluster_holds(int64_t n);
bool dql_in_place(const float *x, int64_t n, const uint8_t *y, const float *y_scale,
    const uint8_t *y_zp);

// gemm_tc.cu / gemm_simt.cu
//
// What the library itself can say about a GEMM beyond the public argument block.
struct GemmCall : omcudaGemmArgs {
  // Row pitch of A in bytes.  More than K only with rows that start 16-byte
  // aligned and hold zeros from K up to the next multiple of 16.
  int64_t lda;
  // The output zero point of the REQUANT tail (one byte of device memory, the
  // output's type); null: y_zp.  Read by the kernel, so that the host never
  // waits for it.
  const uint8_t *y_zp_dev;
  // The host has seen the preparation of B finish: no kernel that may still be running when
  // this GEMM is set up writes it.
  bool b_settled;
  // The kernel behind may be set up while this product runs.  Not for the
  // operators, whose successor may be anything: the blocks of a pass that come early find
  // the SMs of this kernel's last tiles taken and stay together on those that were free.  us
  // of a chain of calls, set up early / at the end (and before dequantize and the passes of
  // more than 16 Mi values overlapped at all):
  //   16384 x 1024 x 4096  linear, DynamicQuantizeLinear                 222 / 203 (211)
  //                        DynamicQuantizeLinear, product, dequantize    199 / 181 (183)
  //   2048 x 1024 x 4096   the same three                                32.2 / 30.4 (31.1)
  //   4096 x 4096 x 4096   linear after linear                           168 / 159 (180)
  //   777 x 1001 x 1537                                                  35.7 / 33.1 (37.2)
  //   700 x 768 x 768                                                    23.5 / 22.9 (25.0)
  // One linear of few rows after another, the same way: 128 x 768 x 768 8.5 / 8.1, 64 x 8192 x 8192
  // 21.6 / 21.1, 61 x 768 x 768 8.0 / 7.7; of one row 768 x 3072 5.8 / 5.6, 4096 x 14336 14.9 / 14.9.
  // For the encoder's, behind which LayerNorm, attention and the quantize pass that folds
  // nothing wait: base 32 x 128 tokens 1400 / 1479, large 32 x 128 3384 / 3527, base 8 x 128 787 /
  // 802 us.
  bool early_next;
  GemmCall()
      : omcudaGemmArgs(), lda(0), y_zp_dev(nullptr), b_settled(false), early_next(false) {}
  explicit GemmCall(const omcudaGemmArgs &a)
      : omcudaGemmArgs(a), lda(a.K), y_zp_dev(nullptr), b_settled(false), early_next(false) {}
};
int gemm_i8(const GemmCall &a, cudaStream_t st);
bool gemm_tc_supported(const GemmCall &a);
// A switch asks for a tile width, epilogue warps or slices of gemm_tc.cu.
bool gemm_tc_forced();
int launch_gemm_tc(const GemmCall &a, cudaStream_t st);
// gemm_few.cu: few rows of A, on the tensor cores.
bool gemm_few_wanted(int64_t M, int64_t N, int64_t K);
// Rows per tile and CTAs per cluster that it would run with.
void gemm_few_plan(int64_t M, int64_t N, int64_t K, int *rows, int *split);
bool gemm_few_supported(const GemmCall &a);
int launch_gemm_few(const GemmCall &a, cudaStream_t st);
int launch_gemm_simt(const GemmCall &a, cudaStream_t st);
// S[i] = a_scale * b_scale[i] / y_scale, the column scales of a QLinearMatMul.
struct RequantScale {
  const float *a_scale, *b_scale, *y_scale;
  int64_t len; // 0: none
  float *S;
};
// Copies an 8-bit [M,K] matrix of any alignment into rows of `pitch` bytes (a
// multiple of 16, dst 16-byte aligned), zero from K on; dst or rowsum may be
// null.  Makes the scales of rq in the same launch.  zp (zp_len bytes, may be
// null): what the sums are for; when all of it is zero they may be left out, and
// rowsum then holds anything.
int launch_repitch(const void *A, int a_signed, int64_t M, int64_t K, int64_t pitch,
    uint8_t *dst, int32_t *rowsum, const RequantScale &rq, cudaStream_t st,
    const void *zp = nullptr, int64_t zp_len = 0);

// linear_rows.cu: DynamicQuantizeLinear, product and DEQUANT tail of up to 16 f32 rows
// in one launch (a: as for gemm_i8, but for its A and what describes it).
bool linear_rows_wanted(int64_t M, int64_t N, int64_t kp);
int linear_rows_groups(int64_t N); // groups of columns per cluster
int launch_linear_rows(const float *x, const GemmCall &a, cudaStream_t st);

// gemm_batched.cu: every product of a MatMulInteger whose B is an activation in
// one launch, operands read as they lie.  Product i (row-major over size[])
// reads A and B at the element offsets its strides give (0 along a broadcast
// dimension) and writes Y at i * M * N.
struct BatchedGemm {
  static constexpr int kMaxDims = 6;
  int M, N, K;
  int dims;
  int64_t size[kMaxDims], a_stride[kMaxDims], b_stride[kMaxDims];
  const void *a_zp; // one value
  int a_zp_len;     // 0 or 1
  const void *b_zp;
  int b_zp_len;     // 0, 1 or N
  // set by gemm_batched_wanted: A takes 16-byte loads everywhere, B 4-byte ones
  int vec_a, vec_b;
  // set by the launcher
  int tiles_m, tiles_n;
  int y_vec; // Y takes stores of 16 bytes (2), of 8 (1), of single values (0)
};
// Whether this kernel is the one for these products on this stream; g has its
// batch dimensions and gets its sizes and alignment.
bool gemm_batched_wanted(const void *A, const void *B, int64_t batch, int64_t M, int64_t N,
    int64_t K, cudaStream_t st, BatchedGemm *g);
int launch_gemm_batched(const void *A, int a_signed, const void *B, int b_signed,
    int32_t *Y, int64_t batch, BatchedGemm g, cudaStream_t st);

// attention_mma.cu
bool attention_mma_supported(const float *Q, const float *K, const float *V,
    const float *out, int64_t dh, int64_t ld_in, int64_t ld_out);
int launch_attention_mma(const float *Q, const float *K, const float *V,
    int64_t B, int64_t S, int64_t heads, int64_t dh, float scale, float *out,
    int64_t ld_in, int64_t ld_out, void *out_range, cudaStream_t st);
// The same kernel on bf16 hi/lo planes (columns of Q, K and V in one row): bit for
// bit what it gives for the fp32 values they were split from.
bool attention_mma_planes_supported(int64_t B, int64_t S, int64_t heads, int64_t dh,
    int64_t ld_planes, int64_t ld_out, const void *hi, const void *lo, const float *out);
int launch_attention_mma_planes(const void *hi, const void *lo, int64_t ld_planes,
    int64_t q_col, int64_t k_col, int64_t v_col, int64_t B, int64_t S, int64_t heads,
    float scale, float *out, int64_t ld_out, void *out_range, cudaStream_t st);

// attention_tc.cu: tcgen05 attention over bf16 hi/lo planes [T, ld_planes]
// (head size 64, sequence a multiple of 128), and the fp32 -> planes split.
bool attention_tc_supported(int64_t B, int64_t S, int64_t heads, int64_t dh,
    int64_t ld_planes, int64_t ld_out, const void *hi, const void *lo,
    const float *out);
int launch_attention_tc(const void *hi, const void *lo, int64_t ld_planes,
    int64_t q_col, int64_t k_col, int64_t v_col, int64_t B, int64_t S,
    int64_t heads, float scale, float *out, int64_t ld_out, void *out_range,
    cudaStream_t st);
int launch_split_bf16(const float *x, int64_t rows, int64_t cols, int64_t ld_x,
    void *hi, void *lo, int64_t ld_p, int64_t col0, cudaStream_t st);

} // namespace omcuda
