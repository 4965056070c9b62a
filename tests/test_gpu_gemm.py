"""GPU parity: MatMulInteger, QLinearMatMul and the fused dynamic-quantized
linear through the C ABI against the CPU oracle.  Bit-exact for int32 / uint8
results; fp32 dequantized outputs are expected bit-exact too and are checked
at the 1e-5 relative tolerance the path's contract states."""
import json
import os

import numpy as np
import pytest

from gpu_util import DevGemm

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
KATS = json.load(open(os.path.join(HERE, "golden", "lit_kats.json")))["cases"]
NP = {"ui8": np.uint8, "i8": np.int8, "i32": np.int32, "f32": np.float32}


def arr(t):
    return None if t is None else np.array(t["data"], dtype=NP[t["dtype"]]).reshape(t["shape"])


def rand8(rng, shape, dt):
    if dt == np.uint8:
        return rng.integers(0, 256, shape, dtype=np.uint8)
    return rng.integers(-128, 128, shape, dtype=np.int8)


@pytest.mark.parametrize("kat", [k for k in KATS if k["op"] == "MatMulInteger"],
                         ids=lambda k: k["name"])
def test_lit_vectors(gpu, kat):
    A, B = arr(kat["A"]), arr(kat["B"])
    want = arr(kat["expected"])
    got = gpu.matmul_integer(A, B, arr(kat["a_zero_point"]), arr(kat["b_zero_point"]))
    assert np.array_equal(got.reshape(want.shape), want)


SHAPES = [(1, 16, 8), (1, 768, 768), (16, 4096, 512), (5, 7, 3), (127, 100, 33),
          (128, 128, 256), (129, 144, 264), (300, 768, 100), (256, 1024, 640),
          (513, 48, 1000), (128, 768, 768)]


@pytest.mark.parametrize("choice", [1, 2], ids=["tcgen05", "simt"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_matmul_integer_kernels(gpu, orc, shape, choice):
    M, K, N = shape
    if choice == 1 and K % 16:
        pytest.skip("tensor-core kernel needs K % 16 == 0; the SIMT kernel covers it")
    rng = np.random.default_rng(M * 31 + K * 7 + N)
    A, B = rand8(rng, (M, K), np.uint8), rand8(rng, (K, N), np.int8)
    az = rng.integers(0, 256, 1, dtype=np.uint8)
    dg = DevGemm(gpu)
    want = orc.matmul_integer_2d(A, B, az, None)
    got = dg.matmul_integer(A, B, az, None, choice)
    assert np.array_equal(got, want), np.argwhere(got != want)[:8]


@pytest.mark.parametrize("choice", [1, 2], ids=["tcgen05", "simt"])
@pytest.mark.parametrize("adt,bdt", [(np.uint8, np.uint8), (np.int8, np.int8),
                                     (np.int8, np.uint8), (np.uint8, np.int8)])
def test_signedness_and_zero_point_forms(gpu, orc, adt, bdt, choice):
    rng = np.random.default_rng(11)
    M, K, N = 130, 160, 72
    A, B = rand8(rng, (M, K), adt), rand8(rng, (K, N), bdt)
    dg = DevGemm(gpu)
    for az, bz in [(None, None), (rand8(rng, 1, adt), None), (None, rand8(rng, 1, bdt)),
                   (rand8(rng, M, adt), rand8(rng, N, bdt)),
                   (rand8(rng, 1, adt), rand8(rng, N, bdt))]:
        want = orc.matmul_integer_2d(A, B, az, bz)
        got = dg.matmul_integer(A, B, az, bz, choice)
        assert np.array_equal(got, want)


@pytest.mark.parametrize("choice", [0, 2], ids=["auto", "simt"])
@pytest.mark.parametrize("adt,bdt", [(np.uint8, np.uint8), (np.int8, np.int8),
                                     (np.int8, np.uint8), (np.uint8, np.int8)])
def test_gemv_shaped_rows_1_to_32(gpu, orc, adt, bdt, choice):
    # The GEMV-shaped kernels (dp4a for one row, mma.sync m16n8k32 with a
    # permuted K order for 2..16) and the hand-over to the tensor-core kernels
    # above 16 rows: ragged M, K (not a multiple of 16 / of the 64-byte block /
    # of a warp's run of blocks) and N (not a multiple of the 16 columns of a
    # block, more blocks than SMs), every signedness and zero-point form.
    rng = np.random.default_rng(41)
    dg = DevGemm(gpu)
    for M, K, N in [(1, 100, 33), (3, 1040, 17), (5, 7, 3), (8, 64, 16), (9, 144, 40),
                    (13, 2000, 70), (16, 4160, 136), (16, 2048, 1000), (2, 16, 8),
                    (7, 1024, 2400), (16, 13312, 48), (23, 1168, 72), (32, 3072, 520)]:
        A, B = rand8(rng, (M, K), adt), rand8(rng, (K, N), bdt)
        for az, bz in [(None, None), (rand8(rng, 1, adt), None),
                       (rand8(rng, M, adt), rand8(rng, N, bdt))]:
            want = orc.matmul_integer_2d(A, B, az, bz)
            got = dg.matmul_integer(A, B, az, bz, choice)
            assert np.array_equal(got, want), (M, K, N, np.argwhere(got != want)[:8])


@pytest.mark.parametrize("M,K,N", [(17, 8192, 256), (100, 8208, 260), (128, 16384, 512),
                                   (129, 8192, 512), (300, 8208, 768), (512, 9216, 1024)])
def test_split_k_shapes(gpu, orc, M, K, N):
    # Up to 512 rows, with few output tiles and K of 8192 or more, the kernels of 128 and
    # 256 rows deal each tile's K loop to several work units (raw partial sums through a
    # workspace, then one reduce pass with the real tail): on single CTAs up to
    # 128 rows, on CTA pairs above.  The raw sums of choice 1 run that way; choice 0 and
    # the operators take the few-rows kernel at these sizes.  All three tails against the
    # oracle, every zero-point form, K not a multiple of the 128-byte K step.  (The real
    # tails of split sums: test_split_k_tails.)
    rng = np.random.default_rng(M + K + N)
    dg = DevGemm(gpu)
    for adt, bdt in [(np.uint8, np.int8), (np.int8, np.uint8)]:
        A, B = rand8(rng, (M, K), adt), rand8(rng, (K, N), bdt)
        for az, bz in [(None, None), (rand8(rng, 1, adt), None),
                       (rand8(rng, M, adt), rand8(rng, N, bdt))]:
            want = orc.matmul_integer_2d(A, B, az, bz)
            for choice in (0, 1):
                got = dg.matmul_integer(A, B, az, bz, choice)
                assert np.array_equal(got, want), (adt, choice, np.argwhere(got != want)[:8])
    # DEQUANT tail (DynamicQuantizeLinear -> MatMulInteger -> Cast -> Mul -> Add)
    X = rng.normal(size=(M, K)).astype(np.float32)
    W = rng.integers(-127, 128, (K, N), dtype=np.int8)
    bias = rng.normal(0, 0.02, N).astype(np.float32)
    ref = orc.dyn_quant_linear(X, W, np.float32(0.0157), bias)
    Y = gpu.dyn_quant_linear(X, W, np.float32(0.0157), None, bias, 0)
    assert Y.tobytes() == ref["Y"].tobytes()
    # REQUANT tail (QLinearMatMul), per-column scales and zero points
    A, B, bs, bz = qlinear_case(rng, (M,), K, N)
    args = (A, np.float32(0.02), np.uint8(128), B, bs, bz, np.float32(0.5), np.uint8(128))
    assert np.array_equal(gpu.qlinear_matmul(*args), orc.qlinear_matmul(*args))


def test_matmul_integer_api_shapes(gpu, orc):
    rng = np.random.default_rng(12)
    # 3-D A times 2-D B (the encoder's broadcast-A form), host and device tensors
    A, B = rand8(rng, (4, 33, 64), np.uint8), rand8(rng, (64, 48), np.int8)
    az = np.array(7, np.uint8)
    want = orc.matmul_integer(A, B, az, None)
    assert np.array_equal(gpu.matmul_integer(A, B, az, None), want)
    assert np.array_equal(gpu.matmul_integer(A, B, az, None, device=True).numpy(), want)
    # equal batch dims on both sides
    A, B = rand8(rng, (3, 17, 32), np.int8), rand8(rng, (3, 32, 20), np.int8)
    assert np.array_equal(gpu.matmul_integer(A, B), orc.matmul_integer(A, B))
    # vector operands
    a, b = rand8(rng, 32, np.uint8), rand8(rng, (32, 9), np.int8)
    assert np.array_equal(gpu.matmul_integer(a, b), orc.matmul_integer(a, b))
    # numpy broadcasting of the batch dimensions (ONNXOps/Math/MatMul.cpp:46-166):
    # size-1 and missing dimensions on either side, a vector against a batch
    for sa, sb in (((4, 1, 5, 16), (3, 16, 7)), ((3, 5, 16), (2, 1, 16, 7)),
                   ((16,), (2, 3, 16, 7)), ((2, 3, 5, 16), (16,)),
                   ((1, 5, 16), (6, 16, 7)), ((2, 3, 5, 16), (2, 3, 16, 7))):
        A, B = rand8(rng, sa, np.uint8), rand8(rng, sb, np.int8)
        az, bz = np.array(9, np.uint8), np.array(-3, np.int8)
        want = orc.matmul_integer(A, B, az, bz)
        got = gpu.matmul_integer(A, B, az, bz)
        assert got.shape == want.shape and np.array_equal(got, want), (sa, sb)
        assert np.array_equal(gpu.matmul_integer(A, B, az, bz, device=True).numpy(), want)
    with pytest.raises(gpu.OmcudaError) as ei:
        gpu.matmul_integer(rand8(rng, (2, 5, 16), np.uint8), rand8(rng, (3, 16, 7), np.int8))
    assert ei.value.code == gpu.EINVAL
    # per-row a zero point, per-column b zero point
    A, B = rand8(rng, (21, 32), np.uint8), rand8(rng, (32, 9), np.uint8)
    az, bz = rand8(rng, 21, np.uint8), rand8(rng, 9, np.uint8)
    assert np.array_equal(gpu.matmul_integer(A, B, az, bz), orc.matmul_integer_2d(A, B, az, bz))


def test_worst_case_magnitude_k14336(gpu, orc):
    # |acc| <= 255 * 128 * 14336 < 2^31: no overflow at the largest K of the sweep
    M, K, N = 64, 14336, 128
    A = np.full((M, K), 255, np.uint8)
    B = np.full((K, N), -128, np.int8)
    B[:, ::2] = 127
    dg = DevGemm(gpu)
    want = orc.matmul_integer_2d(A, B, None, None)
    assert np.array_equal(dg.matmul_integer(A, B, None, None, 1), want)
    assert np.array_equal(dg.matmul_integer(A, B, None, None, 2), want)


def test_full_size_4096_checksums(gpu):
    # Size-independent property at the headline GEMM size: row and column sums
    # of Y equal A @ rowsum(B) and colsum(A) @ B, computed exactly in int64.
    rng = np.random.default_rng(13)
    M = N = K = 4096
    A = rng.integers(0, 256, (M, K), dtype=np.uint8)
    B = rng.integers(-127, 128, (K, N), dtype=np.int8)
    az = np.array([113], np.uint8)
    Y = DevGemm(gpu).matmul_integer(A, B, az, None, 1).astype(np.int64)
    As = A.astype(np.int64) - 113
    assert np.array_equal(Y.sum(1), As @ B.astype(np.int64).sum(1))
    assert np.array_equal(Y.sum(0), As.sum(0) @ B.astype(np.int64))


def qlinear_case(rng, lead, K, N, per_column=True):
    A = rng.integers(0, 256, lead + (K,), dtype=np.uint8)
    B = rng.integers(-127, 128, (K, N), dtype=np.int8)
    bs = rng.uniform(0.001, 0.01, N if per_column else 1).astype(np.float32)
    bz = np.zeros(N if per_column else 1, np.int8)
    return A, B, bs, bz


def test_qlinear_matmul_small_with_wrap(gpu, orc):
    rng = np.random.default_rng(14)
    A, B, bs, bz = qlinear_case(rng, (3, 50), 256, 96)
    bs = (bs * np.float32(16)).astype(np.float32)  # widen so results leave [0,255]
    args = (A, np.float32(0.02), np.uint8(128), B, bs, bz, np.float32(0.5), np.uint8(128))
    want = orc.qlinear_matmul(*args)
    # make sure the case reaches outside [0,255] before the truncation
    acc = (A.reshape(-1, 256).astype(np.int64) - 128) @ B.astype(np.int64)
    pre = np.rint(acc * ((np.float32(0.02) * bs) / np.float32(0.5))[None, :]) + 128
    assert (pre > 255).any() and (pre < 0).any()
    got = gpu.qlinear_matmul(*args)
    assert np.array_equal(got, want)
    bz2 = rng.integers(-5, 6, 96, dtype=np.int8)
    args2 = (A, np.float32(0.02), np.uint8(120), B, bs, bz2, np.float32(0.5), np.uint8(3))
    assert np.array_equal(gpu.qlinear_matmul(*args2), orc.qlinear_matmul(*args2))


def test_qlinear_matmul_int8_output_scalar_scale(gpu, orc):
    rng = np.random.default_rng(15)
    A = rng.integers(-128, 128, (40, 64), dtype=np.int8)
    B = rng.integers(-128, 128, (64, 24), dtype=np.int8)
    args = (A, np.float32(0.1), np.int8(-4), B, np.array([0.05], np.float32),
            np.array([2], np.int8), np.float32(0.7), np.int8(-9))
    assert np.array_equal(gpu.qlinear_matmul(*args), orc.qlinear_matmul(*args))


def test_config2_qlinear_matmul_full_size(gpu, orc):
    # A u8 [32,512,1024], B i8 [1024,4096], per-column b_scale: the whole
    # output on the GPU, a seeded sample of 192 rows against the oracle, plus a
    # byte histogram sanity check that the wrap region is populated.
    rng = np.random.default_rng(42)
    A, B, bs, bz = qlinear_case(rng, (32, 512), 1024, 4096)
    args = (np.float32(0.02), np.uint8(128), B, bs, bz, np.float32(0.5), np.uint8(128))
    got = gpu.qlinear_matmul(A, *args).reshape(-1, 4096)
    rows = rng.choice(32 * 512, 192, replace=False)
    want = orc.qlinear_matmul(A.reshape(-1, 1024)[rows], *args)
    assert np.array_equal(got[rows], want)


def test_config1_dyn_quant_linear(gpu, orc):
    rng = np.random.default_rng(42)
    X = rng.normal(size=(128, 768)).astype(np.float32)
    W = rng.integers(-127, 128, (768, 768), dtype=np.int8)
    bias = rng.normal(0, 0.02, 768).astype(np.float32)
    w_scale = np.float32(0.0157)
    ref = orc.dyn_quant_linear(X, W, w_scale, bias)
    # step by step, as the unfused graph runs
    xq, xs, xz = gpu.dynamic_quantize_linear(X)
    assert np.array_equal(xq, ref["xq"]) and xs == ref["x_scale"] and xz == ref["x_zp"]
    acc = gpu.matmul_integer(xq, W, xz, None)
    assert np.array_equal(acc, ref["acc"])
    # fused
    Y = gpu.dyn_quant_linear(X, W, w_scale, None, bias, 0)
    assert np.allclose(Y, ref["Y"], rtol=1e-5, atol=0)
    assert Y.tobytes() == ref["Y"].tobytes()
    Yd = gpu.dyn_quant_linear(X, W, w_scale, None, bias, 0, device=True).numpy()
    assert Yd.tobytes() == ref["Y"].tobytes()


def test_dyn_quant_linear_forms(gpu, orc):
    rng = np.random.default_rng(16)
    X = rng.normal(size=(2, 37, 96)).astype(np.float32)
    W = rng.integers(-127, 128, (96, 40), dtype=np.int8)
    ref = orc.dyn_quant_linear(X, W, 0.01, None)
    # form 1: (acc * x_scale) * w_scale, two roundings on the tensor
    want1 = orc.dequant_tail(ref["acc"], ref["x_scale"], np.float32(0.01), 1, None)
    got1 = gpu.dyn_quant_linear(X, W, np.float32(0.01), None, None, 1)
    assert got1.tobytes() == want1.tobytes()
    # per-column weight scale
    ws = rng.uniform(0.005, 0.02, 40).astype(np.float32)
    s = (ref["x_scale"] * ws).astype(np.float32)
    want = (ref["acc"].astype(np.float32) * s).astype(np.float32)
    got = gpu.dyn_quant_linear(X, W, ws, None, None, 0)
    assert got.tobytes() == want.tobytes()
    # weight zero point
    wz = np.array(3, np.int8)
    acc = orc.matmul_integer(ref["xq"], W, ref["x_zp"], wz)
    want = orc.dequant_tail(acc, ref["x_scale"] * np.float32(0.01), 0.0, 0, None)
    got = gpu.dyn_quant_linear(X, W, np.float32(0.01), wz, None, 0)
    assert got.tobytes() == want.tobytes()


@pytest.mark.parametrize("K,N", [(4096, 4096), (4096, 14336), (14336, 4096)])
@pytest.mark.parametrize("M", [1, 16, 256, 4096, 16384])
def test_config3_sweep_members(gpu, orc, M, K, N):
    # Every member of the MatMulInteger sweep: DynamicQuantizeLinear over the
    # whole X, then sampled rows of the GEMM and of the dequantized output
    # against the oracle.
    rng = np.random.default_rng(M + K + N)
    X = rng.standard_normal((M, K), dtype=np.float32)
    W = rng.integers(-127, 128, (K, N), dtype=np.int8)
    w_scale = np.float32(0.02 * 4 / 127)
    xq, xs, xz = orc.dynamic_quantize_linear(X)
    Y = gpu.dyn_quant_linear(X, W, w_scale, None, None, 0)
    rows = rng.choice(M, min(M, 48), replace=False)
    acc = orc.matmul_integer_2d(xq[rows], W, xz.reshape(1), None)
    want = orc.dequant_tail(acc, xs * w_scale, 0.0, 0, None)
    assert np.allclose(Y[rows], want, rtol=1e-5, atol=0)
    assert Y[rows].tobytes() == want.tobytes()


def bf16_split(x):
    """hi = bf16(x), lo = bf16(x - hi), round to nearest even, as uint16 bit
    patterns (numpy has no bfloat16)."""
    def to_bf16_bits(f):
        u = f.astype(np.float32).view(np.uint32).astype(np.uint64)
        r = (u + 0x7fff + ((u >> 16) & 1)) >> 16
        return r.astype(np.uint16)
    hi = to_bf16_bits(x)
    hi_f = (hi.astype(np.uint32) << 16).view(np.float32)
    lo = to_bf16_bits((x - hi_f).astype(np.float32))
    return hi, lo


@pytest.mark.parametrize("M,K,N", [(300, 256, 192), (512, 1024, 3072), (33, 64, 72)])
def test_dequant_split_epilogue_equals_split_of_dequant(gpu, M, K, N):
    # The tail that writes bf16 hi/lo planes (operands of the tensor-core
    # attention kernel) must hold exactly the split of the f32 dequant tail.
    from gpu_util import DevGemm
    rng = np.random.default_rng(M + N)
    dg = DevGemm(gpu)
    A = rng.integers(0, 256, (M, K), dtype=np.uint8)
    B = rng.integers(-127, 128, (K, N), dtype=np.int8)
    pb, keep = dg.prepare(B)
    dA = dg.dtensor(A)
    az = dg.dtensor(np.array([131], np.uint8))
    sa = dg.dtensor(np.array([0.013], np.float32))
    sb = dg.dtensor(rng.uniform(0.001, 0.01, N).astype(np.float32))
    bias = dg.dtensor(rng.normal(0, 0.5, N).astype(np.float32))
    g = dg.dev.GemmArgs()
    g.M, g.N, g.K = M, N, K
    g.A, g.a_signed, g.B = dA.data_ptr, 0, pb
    g.a_zp, g.a_zp_len = az.data_ptr, 1
    g.sa, g.sb, g.sb_len, g.bias = sa.data_ptr, sb.data_ptr, N, bias.data_ptr
    g.kernel_choice = dg.dev.KERNEL_TENSOR_CORE
    Y = gpu.Tensor.device_empty((M, N), np.float32)
    g.epilogue, g.Y = dg.dev.EPI_DEQUANT, Y.data_ptr
    dg.dev.gemm_i8(g, dg.stream)
    P = gpu.Tensor.device_empty((2, M, N), np.uint16)
    g.epilogue, g.Y = dg.dev.EPI_DEQUANT_SPLIT, P.data_ptr
    dg.dev.gemm_i8(g, dg.stream)
    y, planes = Y.numpy(), P.numpy()
    gpu.synchronize()
    hi, lo = bf16_split(y)
    assert np.array_equal(planes[0], hi)
    assert np.array_equal(planes[1], lo)
    # and the standalone split kernel writes the same planes
    P2 = gpu.Tensor.device_empty((2, M, N), np.uint16)
    if N % 4 == 0:
        dg.dev.split_bf16(Y.data_ptr, M, N, N, P2.data_ptr, P2.data_ptr + 2 * M * N,
                          N, 0, dg.stream)
        assert np.array_equal(P2.numpy(), planes)


@pytest.mark.parametrize("M,K,N,gelu", [(300, 256, 192, 1), (1024, 1024, 4096, 1),
                                        (33, 64, 72, 0), (515, 512, 1000, 1),
                                        (2600, 512, 1800, 1)])
def test_range_then_quantizing_tails_equal_dequant_then_quantize(gpu, M, K, N, gelu):
    # "linear -> DynamicQuantizeLinear" run as two passes over the product
    # (range only, then quantize while storing uint8) must give the bytes,
    # scale and zero point of the f32 tail followed by the quantize kernel.
    from gpu_util import DevGemm
    rng = np.random.default_rng(M * 7 + N)
    dg = DevGemm(gpu)
    A = rng.integers(0, 256, (M, K), dtype=np.uint8)
    B = rng.integers(-127, 128, (K, N), dtype=np.int8)
    pb, keep = dg.prepare(B)
    dA = dg.dtensor(A)
    az = dg.dtensor(np.array([128], np.uint8))
    sa = dg.dtensor(np.array([0.011], np.float32))
    sb = dg.dtensor(np.array([0.0004], np.float32))
    bias = dg.dtensor(rng.normal(0, 0.5, N).astype(np.float32))
    g = dg.dev.GemmArgs()
    g.M, g.N, g.K = M, N, K
    g.A, g.a_signed, g.B = dA.data_ptr, 0, pb
    g.a_zp, g.a_zp_len = az.data_ptr, 1
    g.sa, g.sb, g.sb_len, g.bias, g.gelu = sa.data_ptr, sb.data_ptr, 1, bias.data_ptr, gelu
    g.kernel_choice = dg.dev.KERNEL_TENSOR_CORE
    ranges = gpu.Tensor.device_empty((4,), np.int32)
    dg.dev.range_init(ranges.data_ptr, 2, dg.stream)
    # reference chain: f32 tail with running range, then the quantize kernel
    Y = gpu.Tensor.device_empty((M, N), np.float32)
    g.epilogue, g.Y, g.out_minmax = dg.dev.EPI_DEQUANT, Y.data_ptr, ranges.data_ptr
    dg.dev.gemm_i8(g, dg.stream)
    q_ref = gpu.Tensor.device_empty((M, N), np.uint8)
    par_ref = gpu.Tensor.device_empty((4,), np.float32)
    dg.dev.quantize_from_range(Y.data_ptr, M * N, ranges.data_ptr, q_ref.data_ptr,
                               par_ref.data_ptr, par_ref.data_ptr + 8,
                               par_ref.data_ptr + 12, dg.stream)
    # two passes over the product, no f32 tensor
    g.epilogue, g.Y, g.out_minmax = dg.dev.EPI_DEQUANT_RANGE, None, ranges.data_ptr + 8
    dg.dev.gemm_i8(g, dg.stream)
    q = gpu.Tensor.device_empty((M, N), np.uint8)
    par = gpu.Tensor.device_empty((4,), np.float32)
    g.epilogue, g.Y, g.out_minmax = dg.dev.EPI_DEQUANT_QUANT, q.data_ptr, None
    g.q_range, g.q_params = ranges.data_ptr + 8, par.data_ptr
    g.q_scale, g.q_zp = par.data_ptr + 8, par.data_ptr + 12
    dg.dev.gemm_i8(g, dg.stream)
    r = ranges.numpy()
    gpu.synchronize()
    assert r[0] == r[2] and r[1] == r[3]
    # slots: scale, zero point as float, y_scale, first byte = y_zero_point
    pw, pw_ref = par.numpy().view(np.uint32), par_ref.numpy().view(np.uint32)
    assert np.array_equal(pw[:3], pw_ref[:3]) and (pw[3] & 0xff) == (pw_ref[3] & 0xff)
    assert np.array_equal(q.numpy(), q_ref.numpy())
    # and the bytes are DynamicQuantizeLinear of the f32 tensor (numpy restatement)
    y = Y.numpy()
    scale = np.float32(np.float32(max(y.max(), 0) - min(y.min(), 0)) / np.float32(255))
    assert par.numpy()[0] == scale


@pytest.mark.parametrize("M,K,N", [(4096, 4096, 4096), (5000, 2048, 4104), (300, 512, 1000),
                                   (2600, 512, 1800), (9300, 256, 2048)])
def test_whole_output_checksums(gpu, orc, M, K, N):
    # Every tile of the output is stored exactly once (the epilogue leaves
    # through TMA stores that clip ragged edges): sampled rows against the
    # oracle and column sums of the whole result against exact integer sums.
    # 4096^3, 2600 x 1800 and 9300 x 2048 end in a round of 256 x 128 half
    # tiles on the 2-CTA kernel (the last two with ragged edges).
    from gpu_util import DevGemm
    rng = np.random.default_rng(K + N)
    A = rng.integers(0, 256, (M, K), dtype=np.uint8)
    B = rng.integers(-127, 128, (K, N), dtype=np.int8)
    dg = DevGemm(gpu)
    rows = np.concatenate([np.arange(0, 40), np.arange(max(M - 300, 40), M, 7)])
    want = orc.matmul_integer_2d(A[rows], B, np.array([117], np.uint8), None)
    Y = dg.matmul_integer(A, B, 117, None, 1)
    assert np.array_equal(Y[rows], want)
    As = A.astype(np.int64) - 117
    assert np.array_equal(Y.astype(np.int64).sum(0), As.sum(0) @ B.astype(np.int64))

@pytest.mark.parametrize("M,K,N,choice", [(300, 256, 192, 1), (260, 512, 1000, 1), (3, 100, 70, 2),
                                          (13, 200, 70, 2), (16, 1040, 136, 0)])
def test_dequant_tail_with_residual(gpu, M, K, N, choice):
    # y = tail(acc) + residual, the onnx.Add of a residual connection folded
    # into the GEMM: one more separately rounded fp32 add, so it must equal
    # the sum of the plain tail's result and the residual bit for bit.
    from gpu_util import DevGemm
    rng = np.random.default_rng(M * N)
    dg = DevGemm(gpu)
    A = rng.integers(0, 256, (M, K), dtype=np.uint8)
    B = rng.integers(-127, 128, (K, N), dtype=np.int8)
    res = rng.normal(0, 1, (M, N)).astype(np.float32)
    pb, keep = dg.prepare(B)
    dA, dres = dg.dtensor(A), dg.dtensor(res)
    az = dg.dtensor(np.array([99], np.uint8))
    sa = dg.dtensor(np.array([0.02], np.float32))
    sb = dg.dtensor(np.array([0.003], np.float32))
    bias = dg.dtensor(rng.normal(0, 0.5, N).astype(np.float32))
    g = dg.dev.GemmArgs()
    g.M, g.N, g.K = M, N, K
    g.A, g.a_signed, g.B = dA.data_ptr, 0, pb
    g.a_zp, g.a_zp_len = az.data_ptr, 1
    g.sa, g.sb, g.sb_len, g.bias = sa.data_ptr, sb.data_ptr, 1, bias.data_ptr
    g.kernel_choice, g.epilogue = choice, dg.dev.EPI_DEQUANT
    Y0 = gpu.Tensor.device_empty((M, N), np.float32)
    g.Y = Y0.data_ptr
    dg.dev.gemm_i8(g, dg.stream)
    Y1 = gpu.Tensor.device_empty((M, N), np.float32)
    g.Y, g.residual = Y1.data_ptr, dres.data_ptr
    dg.dev.gemm_i8(g, dg.stream)
    y0, y1 = Y0.numpy(), Y1.numpy()
    gpu.synchronize()
    assert y1.tobytes() == (y0 + res).astype(np.float32).tobytes()


def check_few_rows(gpu, M, K, N, adt, bdt):
    """The few-rows kernel's sums against the exact product, every tail against the
    128-row tensor-core kernel's, whose arithmetic is the same, bit for bit."""
    rng = np.random.default_rng(M + K + N)
    A, B = rand8(rng, (M, K), adt), rand8(rng, (K, N), bdt)
    dg = DevGemm(gpu)
    D = dg.dev
    zp_a, zp_b = rand8(rng, M, adt), rand8(rng, N, bdt)
    exact = (A.astype(np.float64) - zp_a[:, None]) @ (B.astype(np.float64) - zp_b)  # below 2^53
    assert np.array_equal(dg.matmul_integer(A, B, zp_a, zp_b, 0).astype(np.float64), exact)
    pb, keep = dg.prepare(B)
    f32 = lambda a: dg.dtensor(np.asarray(a, np.float32).reshape(-1))
    dA, az, bz = dg.dtensor(A), dg.dtensor(zp_a[:1]), dg.dtensor(zp_b)
    rs = gpu.Tensor.device_empty((M,), np.int32)
    D.row_sum(dA.data_ptr, int(adt == np.int8), M, K, rs.data_ptr, dg.stream)
    sa, s1, sn = f32(0.013), f32(0.003), f32(rng.uniform(1e-4, 1e-3, N))
    bias, res = f32(rng.normal(0, 0.5, N)), f32(rng.normal(0, 1, M * N))
    for epi, scale, form, extra in (
            (D.EPI_DEQUANT, s1, 0, ()), (D.EPI_DEQUANT, sn, 0, ("bias", "gelu", "range")),
            (D.EPI_DEQUANT, sn, 1, ("bias", "residual", "range", "bz")),
            (D.EPI_DEQUANT_SPLIT, sn, 0, ("bias",)), (D.EPI_REQUANT, sn, 0, ("bz",)),
            (D.EPI_REQUANT, s1, 0, ())):
        out = []
        for choice in (0, D.KERNEL_TENSOR_CORE):
            g = D.GemmArgs()
            g.M, g.N, g.K, g.A, g.a_signed, g.B = M, N, K, dA.data_ptr, int(adt == np.int8), pb
            g.a_zp, g.a_zp_len = az.data_ptr, 1
            if "bz" in extra:
                g.b_zp, g.b_zp_len, g.a_rowsum = bz.data_ptr, N, rs.data_ptr
            g.epilogue, g.scale_form, g.kernel_choice = epi, form, choice
            g.sa, g.sb, g.sb_len = sa.data_ptr, scale.data_ptr, scale.shape[0]
            if "bias" in extra:
                g.bias = bias.data_ptr
            g.gelu = int("gelu" in extra)
            if "residual" in extra:
                g.residual = res.data_ptr
            ranges = gpu.Tensor.device_empty((2,), np.int32)
            if "range" in extra:
                D.range_init(ranges.data_ptr, 1, dg.stream)
                g.out_minmax = ranges.data_ptr
            g.y_zp = 7
            Y = gpu.Tensor.device_empty((M, N), np.uint8 if epi == D.EPI_REQUANT else np.float32)
            g.Y = Y.data_ptr
            D.gemm_i8(g, dg.stream)
            out.append((Y.numpy().tobytes(), ranges.numpy().tobytes() if "range" in extra else b""))
        gpu.synchronize()
        assert out[0] == out[1], (epi, form, extra)


@pytest.mark.parametrize("M,K,N", [
    (17, 16, 8), (17, 128, 128), (32, 144, 129), (33, 1040, 257), (64, 2064, 100), (65, 4096, 130),
    (128, 14336, 72), (129, 640, 1000), (200, 3072, 260), (256, 4112, 3700), (640, 48, 240),
    (16, 3600, 4801), (2, 16384, 4), (48, 64, 12300), (63, 1024, 520)])
@pytest.mark.parametrize("adt,bdt", [(np.uint8, np.int8), (np.int8, np.uint8)])
def test_few_rows_on_the_tensor_cores(gpu, M, K, N, adt, bdt):
    """gemm_few.cu at the edges of its row tiles and of its 128 columns, with slices of K of
    one block and of uneven lengths (tiles of 16 rows, and of 64 in two of them)."""
    check_few_rows(gpu, M, K, N, adt, bdt)


@pytest.mark.parametrize("rows,split,M,K,N", [
    (16, 1, 223, 64, 4), (16, 2, 119, 320, 2), (16, 3, 33, 544, 2), (16, 4, 43, 992, 12),
    (16, 6, 31, 2864, 4), (16, 8, 77, 4656, 4),
    (32, 1, 21, 160, 4136), (32, 2, 17, 336, 490), (32, 3, 17, 608, 839), (32, 4, 594, 4176, 4),
    (32, 6, 457, 4528, 1), (32, 8, 322, 7344, 1),
    (64, 1, 591, 1296, 921), (64, 2, 618, 2544, 389), (64, 3, 575, 2784, 388),
    (64, 4, 599, 4640, 129), (64, 6, 515, 8512, 130), (64, 8, 131, 9264, 385),
    (128, 1, 581, 4208, 1855), (128, 2, 513, 6960, 1028), (128, 3, 500, 6608, 1029),
    (128, 4, 625, 14032, 388), (128, 6, 386, 13488, 386), (128, 8, 71, 9600, 1208)])
@pytest.mark.parametrize("adt,bdt", [(np.uint8, np.int8), (np.int8, np.uint8)])
def test_few_rows_every_cut(gpu, rows, split, M, K, N, adt, bdt):
    """Every row tile with every number of CTAs to its K loop, among them last tiles of one
    to three rows, which most CTAs of the cluster own none of."""
    from omcuda import dev
    assert dev.gemm_few_plan(M, N, K) == (rows, split), "the plan moved: take other sizes"
    check_few_rows(gpu, M, K, N, adt, bdt)


@pytest.mark.parametrize("M,K,N,choice", [
    (17, 8192, 256, 1), (100, 8208, 260, 1), (128, 16384, 512, 1), (129, 8192, 512, 1),
    (300, 8208, 768, 1), (512, 9216, 1024, 1), (100, 14336, 2400, 0), (300, 14336, 2400, 0)])
@pytest.mark.parametrize("adt,bdt", [(np.uint8, np.int8), (np.int8, np.uint8)])
def test_split_k_tails(gpu, M, K, N, choice, adt, bdt):
    """The dequantize and requantize tails behind split sums, on single CTAs (up to 128 rows)
    and on pairs, with bias, per-column scales and zero points, against the same float
    operations on the exact sums, bit for bit; two launches each, the sums and the tail."""
    rng = np.random.default_rng(M + K + N)
    A, B = rand8(rng, (M, K), adt), rand8(rng, (K, N), bdt)
    zp_a, zp_b = rand8(rng, 1, adt), rand8(rng, N, bdt)
    f32 = np.float32
    # sums of at most 255^2 K: exact in float64, below 2^31
    acc = ((A.astype(np.float64) - zp_a) @ (B.astype(np.float64) - zp_b)).astype(f32)
    sb, bias = rng.uniform(1e-4, 1e-3, N).astype(f32), rng.normal(0, 0.5, N).astype(f32)
    dg = DevGemm(gpu)
    D = dg.dev
    pb, keep = dg.prepare(B)
    dA, az, bz = dg.dtensor(A), dg.dtensor(zp_a), dg.dtensor(zp_b)
    rs = gpu.Tensor.device_empty((M,), np.int32)
    D.row_sum(dA.data_ptr, int(adt == np.int8), M, K, rs.data_ptr, dg.stream)
    dsa, dsb, dbias = dg.dtensor(np.array([0.013], f32)), dg.dtensor(sb), dg.dtensor(bias)
    for epi in (D.EPI_DEQUANT, D.EPI_REQUANT):
        g = D.GemmArgs()
        g.M, g.N, g.K, g.A, g.a_signed, g.B = M, N, K, dA.data_ptr, int(adt == np.int8), pb
        g.a_zp, g.a_zp_len = az.data_ptr, 1
        g.b_zp, g.b_zp_len, g.a_rowsum = bz.data_ptr, N, rs.data_ptr
        g.epilogue, g.kernel_choice = epi, choice
        g.sa, g.sb, g.sb_len, g.y_zp = dsa.data_ptr, dsb.data_ptr, N, 7
        if epi == D.EPI_DEQUANT:
            g.bias = dbias.data_ptr
        Y = gpu.Tensor.device_empty((M, N), np.uint8 if epi == D.EPI_REQUANT else f32)
        g.Y = Y.data_ptr
        before = gpu.launch_count()
        D.gemm_i8(g, dg.stream)
        assert gpu.launch_count() - before == 2
        if epi == D.EPI_DEQUANT:
            want = acc * (f32(0.013) * sb) + bias
        else:
            want = (np.rint(acc * sb).astype(np.int64) + 7).astype(np.uint8)
        assert Y.numpy().tobytes() == want.tobytes()
    gpu.synchronize()


@pytest.mark.parametrize("M,K,N", [(700, 768, 768), (2048, 256, 2048), (5000, 128, 4100), (777, 80, 1537)])
def test_passes_behind_a_product(gpu, orc, M, K, N):
    """Products on the tensor cores and the passes that read them, queued without waiting
    (single CTAs and pairs; results on both sides of 16 Mi values): each pass finds its
    product complete, in every one of four rounds over the same buffers."""
    rng = np.random.default_rng(M + N)
    L = gpu.lib()
    B = rand8(rng, (K, N), np.int8)
    As = [rand8(rng, (M, K), np.uint8) for _ in range(4)]
    d = lambda a: gpu.Tensor.from_numpy(np.asarray(a)).to_device()
    dB, dA, sc = d(B), [d(A) for A in As], d(np.float32(0.25))
    L.omcudaRegisterConstant(dB.handle)
    acc, f = gpu.Tensor.device_empty((M, N), np.int32), gpu.Tensor.device_empty((M, N), np.float32)
    q = [gpu.Tensor.device_empty((M, N), np.uint8) for _ in As]
    ys = [(gpu.Tensor.device_empty((), np.float32), gpu.Tensor.device_empty((), np.uint8)) for _ in As]
    for a, y, (s, z) in zip(dA, q, ys):
        L.omcudaMatMulInteger(acc.handle, a.handle, dB.handle, None, None)
        L.omcudaDequantizeLinear(f.handle, acc.handle, sc.handle, None)
        L.omcudaDynamicQuantizeLinear(y.handle, s.handle, z.handle, f.handle)
    gpu.synchronize()
    for A, y, (s, z) in zip(As, q, ys):
        # (sums below 2^24: exact in fp32)
        wy, ws, wz = orc.dynamic_quantize_linear(
            (A.astype(np.float32) @ B.astype(np.float32)) * np.float32(0.25))
        assert s.numpy() == ws and z.numpy() == wz and np.array_equal(y.numpy(), wy)
    L.omcudaForgetConstants()


@pytest.mark.parametrize("K,N", [
    (16, 1), (3000, 5), (2912, 1776), (2913, 1776), (2928, 1777), (1024, 4736), (1025, 4736), (1040, 4737),
    (8192, 4740), (100, 9472), (100, 9473), (2064, 20003)])
@pytest.mark.parametrize("adt,bdt", [(np.uint8, np.int8), (np.int8, np.uint8)])
def test_one_row_at_the_lines_of_its_blocks(gpu, K, N, adt, bdt):
    """One row: blocks of eight, four, two and one warps, on both sides of the lines between
    them (of 148 SMs), with a last group of columns that is short and K that no number of
    warps divides.  Sums against the exact product, the dequantize tail against the same
    float operations, bit for bit."""
    rng = np.random.default_rng(K + N)
    A, B = rand8(rng, (1, K), adt), rand8(rng, (K, N), bdt)
    dg = DevGemm(gpu)
    D = dg.dev
    zp_a, zp_b = rand8(rng, 1, adt), rand8(rng, N, bdt)
    exact = (A.astype(np.float64) - zp_a) @ (B.astype(np.float64) - zp_b)  # below 2^53
    assert np.array_equal(dg.matmul_integer(A, B, zp_a, zp_b, 0).astype(np.float64), exact)
    pb, keep = dg.prepare(B)
    f32 = lambda a: dg.dtensor(np.asarray(a, np.float32).reshape(-1))
    scale, bias = rng.uniform(1e-4, 1e-3, N).astype(np.float32), rng.normal(0, 0.5, N).astype(np.float32)
    dA, sa, sb, db = dg.dtensor(A), f32(0.013), f32(scale), f32(bias)
    Y = gpu.Tensor.device_empty((1, N), np.float32)
    g = D.GemmArgs()
    g.M, g.N, g.K, g.A, g.a_signed, g.B = 1, N, K, dA.data_ptr, int(adt == np.int8), pb
    g.epilogue, g.sa, g.sb, g.sb_len = D.EPI_DEQUANT, sa.data_ptr, sb.data_ptr, N
    g.bias, g.Y = db.data_ptr, Y.data_ptr
    D.gemm_i8(g, dg.stream)
    y = Y.numpy()
    gpu.synchronize()
    acc = (A.astype(np.float64) @ B.astype(np.float64)).astype(np.float32)
    assert y.tobytes() == (acc * (np.float32(0.013) * scale) + bias).tobytes()


@pytest.mark.parametrize("seed", range(16))
def test_random_shapes_against_exact_products(gpu, seed):
    # Ragged shapes drawn at random around the tile sizes of the tensor-core
    # kernels (128 / 256 rows, 64..256 columns, whole and half tiles in the
    # last round, K not a multiple of the 128-byte K step): every output
    # element against the exact integer product (float64 holds it exactly).
    from gpu_util import DevGemm
    rng = np.random.default_rng(1000 + seed)
    M = int(rng.integers(130, 5200))
    N = int(rng.integers(70, 3100))
    K = 16 * int(rng.integers(1, 80))
    a_signed, b_signed = bool(rng.integers(0, 2)), bool(rng.integers(0, 2))
    A = rng.integers(-128 if a_signed else 0, 128 if a_signed else 256, (M, K)).astype(
        np.int8 if a_signed else np.uint8)
    B = rng.integers(-128 if b_signed else 0, 128 if b_signed else 256, (K, N)).astype(
        np.int8 if b_signed else np.uint8)
    za = int(rng.integers(-128 if a_signed else 0, 128 if a_signed else 256))
    dg = DevGemm(gpu)
    Y = dg.matmul_integer(A, B, za, None, 1)
    want = (A.astype(np.float64) - za) @ B.astype(np.float64)
    assert np.array_equal(Y.astype(np.float64), want), (M, N, K, a_signed, b_signed, za)


@pytest.mark.parametrize("seed", range(24))
def test_random_few_rows_long_k_auto_dispatch(gpu, seed):
    # The dispatcher's small-M territory at random: 1..600 rows, K up to 16384,
    # ragged N -- GEMV-shaped kernels (1..16 rows), the few-rows kernel and, for products
    # it leaves, split-K (K >= 8192, few tiles), narrow tiles and the 2-CTA kernel.  Every
    # output element against the exact integer product (float64 holds it exactly), per-row
    # A zero points included.
    from gpu_util import DevGemm
    rng = np.random.default_rng(2000 + seed)
    M = int(rng.choice([1, 2, 3, 7, 8, 15, 16, 17, 31, 64, 100, 128, 129, 200, 256, 300,
                        511, 512, 513, 600]))
    if seed % 3 == 0:
        M = int(rng.integers(1, 601))
    N = int(rng.integers(8, 3000))
    if seed % 2 == 0:
        N = (N + 3) & ~3
    K = 16 * int(rng.integers(1, 1025))
    if seed % 4 == 1:
        K = 16 * int(rng.integers(512, 1025))  # long K
    a_signed, b_signed = bool(rng.integers(0, 2)), bool(rng.integers(0, 2))
    A = rng.integers(-128 if a_signed else 0, 128 if a_signed else 256, (M, K)).astype(
        np.int8 if a_signed else np.uint8)
    B = rng.integers(-128 if b_signed else 0, 128 if b_signed else 256, (K, N)).astype(
        np.int8 if b_signed else np.uint8)
    za = rng.integers(-128 if a_signed else 0, 128 if a_signed else 256,
                      M if seed % 5 == 0 else 1).astype(A.dtype)
    dg = DevGemm(gpu)
    Y = dg.matmul_integer(A, B, za, None, 0)
    want = (A.astype(np.float64) - za.astype(np.float64).reshape(-1, 1)) @ B.astype(np.float64)
    assert np.array_equal(Y.astype(np.float64), want), (M, N, K, a_signed, b_signed)


@pytest.mark.parametrize("lead,M,K,N,adt,bdt", [
    ((1,), 1, 1, 1, np.uint8, np.int8),            # one byte each way
    ((2, 3), 64, 64, 64, np.uint8, np.uint8),      # whole tiles, whole K blocks
    ((2, 3), 61, 61, 64, np.uint8, np.uint8),      # odd K and row pitch
    ((5,), 65, 129, 63, np.int8, np.uint8),        # one past the tile and the K step
    ((3,), 128, 192, 130, np.int8, np.int8),       # N even, not a multiple of 4
    ((2,), 17, 500, 77, np.uint8, np.int8),        # several K steps, ragged last one
    ((), 33, 100, 45, np.uint8, np.uint8),         # one small product, B not a constant
])
def test_batched_b_operand(gpu, orc, lead, M, K, N, adt, bdt):
    # Products whose B is an activation run as one launch on operands as they
    # lie; also with A and B starting at an odd address (views of device
    # buffers), which the word-wise loads have to shift.
    rng = np.random.default_rng(31)
    A, B = rand8(rng, lead + (M, K), adt), rand8(rng, lead + (K, N), bdt)
    az, bz = rand8(rng, (), adt), rand8(rng, (), bdt)
    bzn = rand8(rng, N, bdt)
    for a_zp, b_zp in ((None, None), (az, None), (az, bz), (None, bzn), (az, bzn)):
        want = orc.matmul_integer(A, B, a_zp, b_zp)
        assert np.array_equal(gpu.matmul_integer(A, B, a_zp, b_zp), want), (a_zp, b_zp)
    import torch
    at, bt = (torch.empty(x.size + 3, dtype=torch.uint8, device="cuda") for x in (A, B))
    at[3:] = torch.from_numpy(A.view(np.uint8).reshape(-1)).cuda()
    bt[1:1 + B.size] = torch.from_numpy(B.view(np.uint8).reshape(-1)).cuda()
    av = at[3:].view(torch.int8 if adt == np.int8 else torch.uint8).view(A.shape)
    bv = bt[1:1 + B.size].view(torch.int8 if bdt == np.int8 else torch.uint8).view(B.shape)
    torch.cuda.synchronize()
    got = gpu.matmul_integer(gpu.Tensor.from_cuda_array(av), gpu.Tensor.from_cuda_array(bv), az, bz,
                             device=True)
    assert np.array_equal(got.numpy(), orc.matmul_integer(A, B, az, bz))


def device_view(gpu, x, shift):
    """x on the device, `shift` bytes past an aligned address; and its buffer."""
    import torch
    buf = torch.zeros(x.size + shift, dtype=torch.uint8, device="cuda")
    buf[shift:] = torch.from_numpy(np.ascontiguousarray(x).view(np.uint8).reshape(-1)).cuda()
    torch.cuda.synchronize()
    view = buf[shift:].view(torch.int8 if x.dtype == np.int8 else torch.uint8).view(x.shape)
    return gpu.Tensor.from_cuda_array(view), buf


@pytest.mark.parametrize("shift", [0, 2, 1])
@pytest.mark.parametrize("M,K,N", [(1, 64, 4), (70, 64, 68), (33, 40, 132), (65, 100, 12), (9, 128, 66)])
def test_batched_products_store_widths(gpu, M, K, N, shift):
    # Results leave in 16, 8 or 4 bytes, by N and by where Y starts (in values); the
    # values around Y stay.
    import torch
    rng = np.random.default_rng(M + K + N)
    A, B = rand8(rng, (3, M, K), np.uint8), rand8(rng, (3, K, N), np.uint8)
    a, b = (gpu.Tensor.from_numpy(x).to_device() for x in (A, B))
    az, bz = (gpu.Tensor.from_numpy(np.array(z, np.uint8)).to_device() for z in (131, 120))
    buf = torch.full((4 + 3 * M * N + 4,), -7, device="cuda", dtype=torch.int32)
    y = buf[4 + shift:4 + shift + 3 * M * N].view(3, M, N)
    yt = gpu.Tensor.from_cuda_array(y)
    torch.cuda.synchronize()
    gpu.lib().omcudaMatMulInteger(yt.handle, a.handle, b.handle, az.handle, bz.handle)
    gpu.synchronize()
    got = buf.cpu().numpy()
    want = (A.astype(np.int64) - 131) @ (B.astype(np.int64) - 120)
    assert np.array_equal(got[4 + shift:4 + shift + 3 * M * N].reshape(want.shape), want)
    assert (got[:4 + shift] == -7).all() and (got[4 + shift + 3 * M * N:] == -7).all()


@pytest.mark.parametrize("adt,bdt", [(np.uint8, np.int8), (np.int8, np.uint8)])
@pytest.mark.parametrize("M,K,N", [(1, 101, 70), (9, 101, 70), (16, 96, 33), (17, 101, 64),
                                   (40, 1001, 70), (40, 96, 300)])
def test_registered_weight(gpu, orc, M, K, N, adt, bdt):
    # A weight that is a registered constant takes the prepared path whatever its
    # size: A in aligned rows as it lies, in others read as it lies by the kernels
    # for few rows and copied into aligned rows otherwise, with row sums in that
    # pass or without; the second call uses the prepared form of the first.
    rng = np.random.default_rng(M * K + N)
    A, B = rand8(rng, (M, K), adt), rand8(rng, (K, N), bdt)
    az, bz, bzn = rand8(rng, (), adt), rand8(rng, (), bdt), rand8(rng, N, bdt)
    Bd = gpu.Tensor.from_numpy(B).to_device()
    gpu.lib().omcudaRegisterConstant(Bd.handle)
    try:
        for shift in (0, 1, 3):
            Ad, keep = device_view(gpu, A, shift)
            for a_zp, b_zp in ((None, None), (az, None), (None, bz), (az, bzn)):
                before = gpu.launch_count()
                got = gpu.matmul_integer(Ad, Bd, a_zp, b_zp, device=True).numpy()
                assert gpu.launch_count() > before
                assert np.array_equal(got, orc.matmul_integer(A, B, a_zp, b_zp)), (shift, a_zp, b_zp)
    finally:
        gpu.synchronize()
        gpu.lib().omcudaForgetConstants()


@pytest.mark.parametrize("lead_a,lead_b,M,K,N,constant", [
    # more batch dimensions than the one-launch kernel's argument block holds;
    # eight B slices for 128 products
    ((2, 1, 2, 1, 2, 1, 2), (1, 2, 1, 2, 1, 2, 1), 5, 33, 7, False),
    ((2, 1, 2, 1, 2, 1, 2), (1, 2, 1, 2, 1, 2, 1), 19, 33, 16, False),
    ((3,), (3,), 20, 48, 24, True),          # a batched weight
    ((2, 3), (3,), 4, 31, 9, True),          # ... shared by the outer dimension
    ((2,), (2,), 1024, 1025, 1032, False),   # products too large for mma.sync
])
def test_products_one_after_another(gpu, orc, lead_a, lead_b, M, K, N, constant):
    # The prepared path of a batched B: a loop over the products, A slices at
    # whatever address they start, B slices prepared once each.
    rng = np.random.default_rng(M * K + N)
    A, B = rand8(rng, lead_a + (M, K), np.uint8), rand8(rng, lead_b + (K, N), np.int8)
    Bd = gpu.Tensor.from_numpy(B).to_device()
    if constant:
        gpu.lib().omcudaRegisterConstant(Bd.handle)
    try:
        for a_zp, b_zp in ((None, None), (np.array(9, np.uint8), None),
                           (np.array(9, np.uint8), rand8(rng, N, np.int8))):
            before = gpu.launch_count()
            got = gpu.matmul_integer(gpu.Tensor.from_numpy(A).to_device(), Bd, a_zp, b_zp, device=True)
            assert gpu.launch_count() - before > 1
            assert np.array_equal(got.numpy(), orc.matmul_integer(A, B, a_zp, b_zp))
    finally:
        gpu.synchronize()
        gpu.lib().omcudaForgetConstants()


@pytest.mark.parametrize("batch,M,K,N,one", [
    (1, 1, 16384, 64, True), (1, 1, 16400, 64, False), (1, 1, 16400, 68, True),  # whole words
    (1, 17, 2047, 64, True), (1, 17, 2049, 64, False),      # A in single bytes
    (1, 16, 2049, 64, True),                                # ... of which there are few
    (1, 1, 384, 63, True), (1, 1, 385, 63, False),          # B in single bytes
    (2, 1, 2048, 63, True), (2, 1, 2049, 63, False), (2, 1, 4099, 64, True),
    (3, 1, 16401, 63, True),                                # from three products on
    (1, 1, 65535 * 64 + 1, 1, True),                        # B cannot be prepared
])
def test_which_products_run_in_one_launch(gpu, orc, batch, M, K, N, one):
    # A product whose B is no constant goes to the one-launch kernel where that
    # is the faster way: both sides of each line of the rule.
    rng = np.random.default_rng(K + N)
    lead = (batch,) if batch > 1 else ()
    A, B = rand8(rng, lead + (M, K), np.uint8), rand8(rng, lead + (K, N), np.int8)
    az, bz = rand8(rng, (), np.uint8), rand8(rng, (), np.int8)
    t = [gpu.Tensor.from_numpy(x).to_device() for x in (A, B, az, bz)]
    before = gpu.launch_count()
    got = gpu.matmul_integer(*t, device=True)
    assert (gpu.launch_count() - before == 1) == one
    assert np.array_equal(got.numpy(), orc.matmul_integer(A, B, az, bz))


def test_captured_product_needs_no_pool(gpu, orc):
    # A product with a long K, which would go to the prepared path, stays one launch
    # on the operands as they lie while its stream is being captured: a replay
    # reads what the tensors hold then and writes nothing but Y.
    import torch
    M, K, N = 3, 4099, 63
    rng = np.random.default_rng(37)
    a, b = (torch.empty(s, dtype=torch.uint8, device="cuda") for s in ((M, K), (K, N)))
    y = torch.zeros((M, N), dtype=torch.int32, device="cuda")
    az, bz = (torch.tensor(v, dtype=torch.uint8, device="cuda") for v in (7, 200))
    t = [gpu.Tensor.from_cuda_array(x) for x in (y, a, b, az, bz)]
    call = [x.handle for x in t]
    L = gpu.lib()
    before = gpu.launch_count()
    L.omcudaMatMulInteger(*call)
    assert gpu.launch_count() - before > 1
    gpu.check()
    # (a short K loads the one-launch kernel outside the capture)
    gpu.matmul_integer(rand8(rng, (M, 301), np.uint8), rand8(rng, (301, N), np.uint8),
                       np.array(7, np.uint8), np.array(200, np.uint8))
    gpu.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    try:
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            L.omcudaSetStream(stream.cuda_stream)
            before = gpu.launch_count()
            L.omcudaMatMulInteger(*call)
            assert gpu.launch_count() - before == 1
    finally:
        L.omcudaSetStream(None)
    gpu.check()
    for _ in range(2):
        A, B = rand8(rng, (M, K), np.uint8), rand8(rng, (K, N), np.uint8)
        a.copy_(torch.from_numpy(A))
        b.copy_(torch.from_numpy(B))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        want = orc.matmul_integer(A, B, np.array(7, np.uint8), np.array(200, np.uint8))
        assert np.array_equal(y.cpu().numpy(), want)


@pytest.mark.parametrize("M,K,N", [(1, 2, (1 << 27) + 4),  # 28 rows of B are beyond 2^31
                                   (1, 17 << 21, 1)])       # 63 rows of A are
def test_batched_b_operand_offsets(gpu, M, K, N):
    # The offsets of a tile's rows that do not exist would not fit 32 bits.
    import torch
    g = torch.Generator(device="cuda").manual_seed(35)
    a = torch.randint(0, 256, (3, M, K), device="cuda", generator=g, dtype=torch.uint8)
    b = torch.randint(0, 256, (3, K, N), device="cuda", generator=g, dtype=torch.uint8)
    torch.cuda.synchronize()
    y = gpu.matmul_integer(gpu.Tensor.from_cuda_array(a), gpu.Tensor.from_cuda_array(b), device=True)
    got = torch.as_tensor(y, device="cuda")
    for i in range(3):
        if N == 1:
            want = (a[i, 0].int() * b[i, :, 0].int()).sum(dtype=torch.int64).to(torch.int32)
            assert got[i].item() == want.item()
        else:
            assert torch.equal(got[i, 0], (a[i].reshape(K, 1).int() * b[i].int()).sum(0, dtype=torch.int32))


@pytest.mark.parametrize("M,K,N,wdt", [
    (1, 17, 5, np.uint8), (16, 257, 33, np.int8),   # GEMV-shaped kernels, padded rows
    (17, 15, 64, np.uint8),                         # less than one 16-byte chunk of K
    (33, 129, 63, np.int8),                         # one past a K step, ragged store
    (300, 1001, 257, np.uint8),                     # several tiles each way
    (2100, 143, 300, np.int8),                      # CTA pairs
])
def test_ragged_k_and_n(gpu, orc, M, K, N, wdt):
    # K that is no multiple of 16: the quantized rows (and an 8-bit A) are laid
    # out with a padded pitch for the tensor-core kernels.  N that is none:
    # results leave row by row instead of through TMA stores.
    rng = np.random.default_rng(32)
    X = rng.normal(size=(M, K)).astype(np.float32)
    W, wz, bias = rand8(rng, (K, N), wdt), rand8(rng, (), wdt), rng.normal(size=N).astype(np.float32)
    ref = orc.dyn_quant_linear(X, W, 0.01, bias) if wdt == np.int8 else None
    if ref is not None:
        assert gpu.dyn_quant_linear(X, W, np.float32(0.01), None, bias).tobytes() == ref["Y"].tobytes()
    xq, xs, xz = orc.dynamic_quantize_linear(X)
    acc = orc.matmul_integer(xq, W, xz, wz)
    want = orc.dequant_tail(acc, xs * np.float32(0.01), 0.0, 0, bias)
    assert gpu.dyn_quant_linear(X, W, np.float32(0.01), wz, bias).tobytes() == want.tobytes()
    # per-row A zero points take the prepared path whatever the size
    azn, bzn = rand8(rng, M, np.uint8), rand8(rng, N, wdt)
    assert np.array_equal(gpu.matmul_integer(xq, W, azn, bzn), orc.matmul_integer_2d(xq, W, azn, bzn))
    if wdt == np.int8:
        bs = rng.uniform(0.001, 0.01, N).astype(np.float32)
        args = (xq, np.float32(0.02), np.uint8(128), W, bs, bzn, np.float32(0.5), np.uint8(7))
        assert np.array_equal(gpu.qlinear_matmul(*args), orc.qlinear_matmul(*args))


@pytest.mark.parametrize("wdt,zp", [(np.int8, None), (np.uint8, 131)])
@pytest.mark.parametrize("M,K,N", [(2, 8192, 9000), (15, 2176, 15400), (4, 4096, 14337), (3, 5000, 10000)])
def test_few_rows_of_many_column_groups(gpu, M, K, N, wdt, zp):
    # Sizes that a cluster would take in several column groups: quantize and product by
    # themselves, one launch (no scratch) while the stream is being captured, and the same
    # bits: the zero point of the weight is one value here.
    import torch
    rng = np.random.default_rng(M + N)
    x = torch.from_numpy(rng.normal(0.1, 1, size=(M, K)).astype(np.float32)).cuda()
    w = torch.from_numpy(rand8(rng, (K, N), wdt)).cuda()
    ws, y = torch.tensor(0.0157, device="cuda"), torch.zeros((2, M, N), device="cuda")
    z = torch.tensor(zp, dtype=torch.uint8, device="cuda") if zp else None
    T = gpu.Tensor.from_cuda_array
    t = [T(x), T(w), T(ws)] + ([T(z)] if zp else [])
    ys = [T(y[0]), T(y[1])]
    L = gpu.lib()
    L.omcudaRegisterConstant(t[1].handle)
    args = [a.handle for a in t] + ([] if zp else [None]) + [None, 0]
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    try:
        L.omcudaSetStream(stream.cuda_stream)
        for _ in range(2):
            before = gpu.launch_count()
            L.omcudaDynQuantLinear(ys[0].handle, *args)
            assert gpu.launch_count() - before >= 2
        gpu.check()
        gpu.synchronize()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            before = gpu.launch_count()
            L.omcudaDynQuantLinear(ys[1].handle, *args)
            assert gpu.launch_count() - before == 1
        gpu.check()
        graph.replay()
        torch.cuda.synchronize()
        got = y.cpu().numpy()
        assert got[0].tobytes() == got[1].tobytes() and np.abs(got[0]).max() > 0
    finally:
        L.omcudaSetStream(None)
        torch.cuda.synchronize()
        L.omcudaForgetConstants()


@pytest.mark.parametrize("rest", [1, 7, 8, 9, 24, 25, 31])
@pytest.mark.parametrize("N", [259, 1537])
@pytest.mark.parametrize("tail", ["i32", "dequant", "requant"])
def test_ragged_rows_leave_eight_together(gpu, rest, N, tail):
    # The last 32-row block of a tile has `rest` rows, the last 32 columns 3 or 1: whole
    # results, and nothing before or behind them.
    M, K, pad = 672 + rest, 64, 64
    rng = np.random.default_rng(rest + N)
    A, B = rand8(rng, (M, K), np.uint8), rand8(rng, (K, N), np.int8)
    dg = DevGemm(gpu)
    D = dg.dev
    pb, keep = dg.prepare(B)
    dA = dg.dtensor(A)
    esize = 1 if tail == "requant" else 4
    Y = dg.dtensor(np.full((M * N + 2 * pad) * esize, 0x5a, np.uint8))
    S = dg.dtensor(np.full(1, 0.03125, np.float32))
    g = D.GemmArgs()
    g.M, g.N, g.K, g.A, g.a_signed, g.B = M, N, K, dA.data_ptr, 0, pb
    g.Y = Y.data_ptr + pad * esize
    g.sa = g.sb = S.data_ptr
    g.sb_len = 1
    g.kernel_choice = D.KERNEL_TENSOR_CORE
    g.epilogue = {"i32": D.EPI_I32, "dequant": D.EPI_DEQUANT, "requant": D.EPI_REQUANT}[tail]
    if tail == "requant":
        g.sa = None
    D.gemm_i8(g, dg.stream)
    out = Y.numpy()
    gpu.synchronize()
    acc = A.astype(np.int64) @ B.astype(np.int64)
    want = {"i32": acc.astype(np.int32), "dequant": (acc * 2.0 ** -10).astype(np.float32),
            "requant": np.rint(acc * 2.0 ** -5).astype(np.int64).astype(np.uint8)}[tail]
    assert out[pad * esize:-pad * esize].tobytes() == want.tobytes()
    assert (out[:pad * esize] == 0x5a).all() and (out[-pad * esize:] == 0x5a).all()


@pytest.mark.parametrize("ydt", [np.uint8, np.int8])
@pytest.mark.parametrize("M,K,N,per_column", [(1, 64, 40, False), (9, 48, 33, True),
                                              (40, 100, 300, True), (300, 64, 512, False)])
def test_qlinear_parameters_on_the_device(gpu, orc, ydt, M, K, N, per_column):
    # y_zero_point is read by the kernels' tails and the column scales are made
    # in the row-sum pass; every kernel family, both output types, host and
    # device parameters alike.
    rng = np.random.default_rng(33)
    A, B = rand8(rng, (M, K), np.uint8), rand8(rng, (K, N), np.int8)
    bs = rng.uniform(0.001, 0.01, N if per_column else ()).astype(np.float32)
    bz = rand8(rng, N if per_column else (), np.int8)
    yz = np.asarray(-77 if ydt == np.int8 else 200, ydt)
    args = (A, np.float32(0.02), np.uint8(128), B, bs, bz, np.float32(0.5), yz)
    want = orc.qlinear_matmul(*args)
    assert np.array_equal(gpu.qlinear_matmul(*args), want)
    assert np.array_equal(gpu.qlinear_matmul(*args, device=True).numpy(), want)


@pytest.mark.parametrize("M,K,N", [(1, 64, 255), (1, 33, 256), (8, 64, 257), (9, 40, 5000),
                                   (70, 64, 40)])
def test_qlinear_scales_beside_row_sums(gpu, orc, M, K, N):
    # One launch makes the row sums (8 rows a block) and the column scales (256 a
    # block): more blocks of either, and the edges of both.
    rng = np.random.default_rng(M + N)
    A, B, bs, _ = qlinear_case(rng, (M,), K, N)
    bz = rand8(rng, N, np.int8)
    args = (A, np.float32(0.02), np.uint8(128), B, bs, bz, np.float32(0.5), np.uint8(11))
    assert np.array_equal(gpu.qlinear_matmul(*args, device=True).numpy(), orc.qlinear_matmul(*args))


@pytest.mark.parametrize("scale", [0.9, 70.0, 3e7])
def test_qlinear_large_results(gpu, orc, scale):
    # Results around and beyond 2^22 (and 2^31, where the conversion saturates):
    # the tail's one-addition rounding hands those to the separate instructions.
    rng = np.random.default_rng(34)
    A, B = rand8(rng, (200, 512), np.uint8), rand8(rng, (512, 320), np.int8)
    bs = (rng.uniform(0.5, 1.5, 320) * scale).astype(np.float32)
    args = (A, np.float32(1.0), np.uint8(128), B, bs, np.zeros(320, np.int8), np.float32(1.0),
            np.uint8(9))
    x = np.abs((A.astype(np.int64) - 128) @ B.astype(np.int64)) * bs[None, :].astype(np.float64)
    inside = x < 2**31 - 256     # beyond it the C conversion of the oracle is undefined
    got, want = gpu.qlinear_matmul(*args), orc.qlinear_matmul(*args)
    assert np.array_equal(got[inside], want[inside]) and inside.any()
    assert (x > 2**22).any() or scale < 1


@pytest.mark.parametrize("m,k,n", [(40, 64, 128), (300, 192, 144), (9, 1024, 96), (150, 77, 133)])
@pytest.mark.parametrize("zeros", ["all", "chunks", "none"])
@pytest.mark.parametrize("yt", [np.uint8, np.int8])
def test_weight_zero_points_partly_zero(gpu, orc, m, k, n, zeros, yt):
    """Zero points of the weight that are all zero, zero in whole runs of 32 columns
    (which the tails skip), or nowhere; output zero points at the end of their type."""
    rng = np.random.default_rng(m + k + n)
    a = rng.integers(0, 256, (m, k)).astype(np.uint8)
    b = rng.integers(-128, 128, (k, n)).astype(np.int8)
    bz = np.zeros(n, np.int8) if zeros == "all" else rng.integers(1, 100, n).astype(np.int8)
    if zeros == "chunks":
        bz[32:96] = 0
    bs = (rng.random(n) * 0.009 + 0.001).astype(np.float32)
    yz = yt(np.iinfo(yt).max)
    args = (a, np.float32(0.02), np.uint8(131), b, bs, bz, np.float32(0.37), yz)
    want = orc.qlinear_matmul(*args)
    assert np.array_equal(gpu.qlinear_matmul(*args), want)
    assert np.array_equal(gpu.qlinear_matmul(*args, device=True).numpy(), want)


@pytest.mark.parametrize("k,n", [(1, 1), (3, 5), (16, 4), (63, 65), (64, 64), (65, 130), (200, 67),
                                 (130, 256)])
@pytest.mark.parametrize("signed", [False, True])
def test_prepared_weight(gpu, k, n, signed):
    """The K-major copy of a weight, its zero padding and its column sums."""
    import torch
    from omcuda import dev
    rng = np.random.default_rng(k * 300 + n)
    w = rng.integers(0, 256, (k, n)).astype(np.uint8)
    nbytes, kp = dev.prepared_b_bytes(k, n)
    for shift in (0, 1):
        src = torch.zeros(k * n + 1, dtype=torch.uint8, device="cuda")
        src[shift:shift + k * n] = torch.from_numpy(w.ravel()).cuda()
        bt = torch.full((nbytes,), 255, dtype=torch.uint8, device="cuda")
        cs = torch.empty(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        dev.prepare_b(src.data_ptr() + shift, int(signed), k, n, bt.data_ptr(), cs.data_ptr(), None)
        torch.cuda.synchronize()
        got = bt.cpu().numpy().reshape(n, kp)
        assert np.array_equal(got[:, :k], w.T) and not got[:, k:].any()
        v = w.view(np.int8) if signed else w
        assert np.array_equal(cs.cpu().numpy(), v.astype(np.int64).sum(0))


@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (1, 15, 63), (2, 64, 64), (16, 512, 65), (16, 513, 200), (3, 1040, 128),
                                   (7, 4099, 130), (16, 8200, 96), (2, 16001, 2100), (3, 5461, 33), (2, 500, 18000),
                                   (16, 1024, 2496), (4, 768, 3072)])
@pytest.mark.parametrize("wt,per_column", [(np.int8, False), (np.uint8, True), (np.uint8, False)])
@pytest.mark.parametrize("form", [0, 1])
def test_linear_of_few_rows(gpu, orc, m, k, n, wt, per_column, form):
    """Up to 16 rows in one launch, K split over a cluster: slices that are empty, that
    end inside a 64-byte block, several column groups per cluster, and sizes that are
    left to the separate kernels (which is which: the test below)."""
    rng = np.random.default_rng(m * 31 + k + n)
    x = rng.normal(0.2, 2, size=(m, k)).astype(np.float32)
    w = rng.integers(-127, 128, (k, n)).astype(np.int8) if wt == np.int8 else \
        rng.integers(0, 256, (k, n)).astype(np.uint8)
    zp = None if wt == np.int8 else (rng.integers(0, 256, n).astype(np.uint8) if per_column
                                     else np.array(131, np.uint8))
    ws = (rng.random(n) * 0.009 + 0.001).astype(np.float32) if per_column else np.float32(0.0157)
    bias = rng.normal(size=n).astype(np.float32) if m % 2 else None
    xq, xs, xz = orc.dynamic_quantize_linear(x)
    xi = (xq.astype(np.float64) - float(xz))
    wi = w.astype(np.float64) - (0.0 if zp is None else zp.astype(np.float64))
    f = (xi @ wi).astype(np.int64).astype(np.float32)  # exact: |sum| < 2^53
    want = f * (np.float32(xs) * ws) if form == 0 else (f * np.float32(xs)) * ws
    want = want.astype(np.float32)
    if bias is not None:
        want = want + bias
    for device in (False, True):
        got = gpu.dyn_quant_linear(x, w, ws, zp, bias, form, device=device)
        got = got.numpy() if device else got
        assert got.tobytes() == want.astype(np.float32).tobytes()


@pytest.mark.parametrize("m,k,n,at", [(2, 1024, 1024, 0), (8, 1024, 1024, 0), (16, 512, 512, 0), (4, 2048, 1000, 0),
                                      (4, 1000, 1500, 500), (4, 1000, 1500, 3999), (3, 64, 64, 191)])
def test_linear_onto_its_input(gpu, orc, m, k, n, at):
    """Y in the memory of X, from element `at` of X on: X is read completely before Y
    is written."""
    import torch
    rng = np.random.default_rng(m + k + n)
    x = rng.normal(0.2, 2, size=(m, k)).astype(np.float32)
    w = rng.integers(-127, 128, (k, n)).astype(np.int8)
    xq, xs, xz = orc.dynamic_quantize_linear(x)
    acc = (xq.astype(np.int64) - int(xz)) @ w.astype(np.int64)
    want = acc.astype(np.float32) * (np.float32(xs) * np.float32(0.0157))
    wd = gpu.Tensor.from_numpy(w).to_device()
    ws = gpu.Tensor.from_numpy(np.array(0.0157, np.float32)).to_device()
    L = gpu.lib()
    L.omcudaRegisterConstant(wd.handle)
    try:
        for inside in (False, True, True):
            buf = torch.zeros(at + 2 * m * max(k, n), device="cuda")
            buf[:m * k] = torch.from_numpy(x.ravel()).cuda()
            first = at if inside else m * k
            xd = gpu.Tensor.from_cuda_array(buf[:m * k].view(m, k))
            yd = gpu.Tensor.from_cuda_array(buf[first:first + m * n].view(m, n))
            torch.cuda.synchronize()
            before = gpu.launch_count()
            L.omcudaDynQuantLinear(yd.handle, xd.handle, wd.handle, ws.handle, None, None, 0)
            gpu.synchronize()
            launches = gpu.launch_count() - before
            got = buf[first:first + m * n].cpu().numpy().reshape(m, n)
            assert got.tobytes() == want.astype(np.float32).tobytes()
        assert launches == 2  # (quantize and product; the weight is prepared by now)
    finally:
        gpu.synchronize()
        L.omcudaForgetConstants()


@pytest.mark.parametrize("m,k,n,one", [
    (2, 64, 64, True), (16, 1009, 65, True), (3, 1040, 128, True), (16, 1024, 1984, True),
    (15, 2176, 15400, True),   # all five words of x that a thread can hold
    (2, 16001, 2100, True), (2, 8192, 9000, True),  # several column groups per cluster
    (1, 64, 64, False), (17, 64, 64, False), (24, 1001, 130, False), (4, 768, 3072, False),
    (16, 1040, 96, False), (4, 8208, 5000, False), (16, 2048, 400, False)])
@pytest.mark.parametrize("data", ["normal", "zero", "negative", "nan", "inf", "tiny"])
def test_linear_of_few_rows_values(gpu, orc, m, k, n, one, data):
    """One launch for a prepared weight or not, by the sizes, and either way the values
    of the separate operators: activations that quantize with a scale of zero or
    beyond the divide-free range, infinities and NaNs, rows that do not start on 16
    bytes, and the modes without zero point and with the reciprocal."""
    import torch
    rng = np.random.default_rng(m * 31 + k + n)
    x = rng.normal(0.2, 2, size=(m, k)).astype(np.float32)
    if data == "zero":
        x[:] = 0
    elif data == "negative":
        x = -np.abs(x) - 1
    elif data == "nan":
        x.ravel()[::61] = np.nan
    elif data == "inf":
        x.ravel()[m * k // 2] = np.inf
    elif data == "tiny":
        x *= np.float32(1e-35)
    w = rng.integers(0, 256, (k, n)).astype(np.uint8)
    zp = rng.integers(0, 256, n).astype(np.uint8)
    ws = (rng.random(n) * 0.009 + 0.001).astype(np.float32)
    wi = (w.astype(np.float64) - zp)
    t = [gpu.Tensor.from_numpy(a).to_device() for a in (w, ws, zp)]
    L = gpu.lib()
    L.omcudaRegisterConstant(t[0].handle)
    try:
        for mode, shift in ((0, 0), (0, 1), (1, 0), (2, 0), (3, 0)):
            buf = torch.zeros(m * k + 1, device="cuda")
            buf[shift:shift + m * k] = torch.from_numpy(x.ravel()).cuda()
            y = torch.zeros((m, n), device="cuda")
            xd = gpu.Tensor.from_cuda_array(buf[shift:shift + m * k].view(m, k))
            yd = gpu.Tensor.from_cuda_array(y)
            torch.cuda.synchronize()
            orc.L.orc_set_quant_mode(mode)
            L.omcudaSetQuantizationMode(mode)
            try:
                xq, xs, xz = orc.dynamic_quantize_linear(x)
                for _ in range(2):
                    before = gpu.launch_count()
                    L.omcudaDynQuantLinear(yd.handle, xd.handle, *[a.handle for a in t], None, 0)
                    launches = gpu.launch_count() - before
            finally:
                L.omcudaSetQuantizationMode(0)
                orc.L.orc_set_quant_mode(0)
            gpu.synchronize()
            assert (launches == 1) == one
            acc = ((xq.astype(np.float64) - float(xz)) @ wi).astype(np.int64)  # exact: below 2^53
            with np.errstate(invalid="ignore"):
                want = acc.astype(np.float32) * (np.float32(xs) * ws)
            assert np.array_equal(y.cpu().numpy(), want.astype(np.float32), equal_nan=True), (mode, shift)
    finally:
        gpu.synchronize()
        L.omcudaForgetConstants()
