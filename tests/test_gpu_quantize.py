"""GPU parity: DynamicQuantizeLinear / QuantizeLinear / DequantizeLinear through
the C ABI against the CPU oracle.  Bit-exact for the uint8 tensor, the scale
and the zero point."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check_dql(gpu, orc, x, device=False):
    want_y, want_s, want_z = orc.dynamic_quantize_linear(x)
    if device:
        y, s, z = gpu.dynamic_quantize_linear(x, device=True)
        y, s, z = y.numpy(), s.numpy(), z.numpy()
    else:
        y, s, z = gpu.dynamic_quantize_linear(x)
    assert s.tobytes() == want_s.tobytes(), (s, want_s)
    assert int(z) == int(want_z)
    assert y.shape == want_y.shape
    assert np.array_equal(y, want_y), np.flatnonzero(y.ravel() != want_y.ravel())[:10]


def test_config1_activation(gpu, orc):
    x = np.random.default_rng(42).normal(size=(128, 768)).astype(np.float32)
    check_dql(gpu, orc, x)
    check_dql(gpu, orc, x, device=True)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 33, 255, 1023, 1025, 4097, 100003])
def test_ragged_sizes(gpu, orc, n):
    x = np.random.default_rng(n).normal(0, 3, size=n).astype(np.float32)
    check_dql(gpu, orc, x)


def test_rank0_and_rank4(gpu, orc):
    check_dql(gpu, orc, np.array(2.5, np.float32))
    check_dql(gpu, orc, np.random.default_rng(1).normal(size=(2, 3, 5, 7)).astype(np.float32))


def test_edge_values(gpu, orc):
    check_dql(gpu, orc, np.zeros(1000, np.float32))                  # scale 0 -> NaN path
    check_dql(gpu, orc, np.linspace(1, 9, 777, dtype=np.float32))    # all positive
    check_dql(gpu, orc, -np.linspace(1, 9, 777, dtype=np.float32))   # all negative
    x = np.random.default_rng(3).normal(size=4099).astype(np.float32)
    x[[0, 100, 4098]] = np.nan
    check_dql(gpu, orc, x)                                           # NaN ignored by min/max
    x = np.random.default_rng(4).normal(size=513).astype(np.float32)
    x[7], x[9] = 1e30, -1e30
    check_dql(gpu, orc, x)                                           # huge range
    check_dql(gpu, orc, np.array([-0.0, 0.0, 1e-40, -1e-40, 1.0], np.float32))  # denormals


def test_exact_ties(gpu, orc):
    # range [-127.5, 127.5] -> scale 1.0, zero point 128 (127.5 rounds to even):
    # every k + 0.5 is an exact tie of x / scale.
    x = np.concatenate([np.arange(-127, 127, dtype=np.float32) + 0.5,
                        np.array([-127.5, 127.5], np.float32),
                        np.arange(-127, 128, dtype=np.float32)])
    _, s, _ = orc.dynamic_quantize_linear(x)
    assert s == 1.0
    check_dql(gpu, orc, x)


def test_values_crowded_around_ties(gpu, orc):
    # The kernel avoids the divide on its common path and falls back to the
    # exact divide near a rounding tie: crowd the input around ties, at every
    # magnitude of the quantized range and at offsets from far below to far
    # above the fallback threshold.
    rng = np.random.default_rng(9)
    for lo, hi in ((-3.7, 5.1), (-1000.0, 0.3), (-1e-3, 2e-3), (0.0, 7.77)):
        scale = np.float32((np.float32(hi) - np.float32(lo)) / np.float32(255))
        k = rng.integers(-300, 300, size=400000).astype(np.float32)
        off = rng.choice([0.0, 1e-7, -1e-7, 3e-6, -3e-6, 1e-4, -1e-4, 9e-4, -9e-4,
                          2e-3, -2e-3, 0.25], size=k.size).astype(np.float32)
        x = ((k + np.float32(0.5) + off) * scale).astype(np.float32)
        x = np.clip(x, np.float32(lo), np.float32(hi))
        x[0], x[1] = np.float32(lo), np.float32(hi)      # pins the range
        check_dql(gpu, orc, x)


def test_larger_than_l2(gpu, orc):
    # 48 Mi floats = 192 MiB > the 126 MB L2: the quantize pass re-reads HBM.
    x = np.random.default_rng(5).normal(size=48 * 1024 * 1024).astype(np.float32)
    check_dql(gpu, orc, x, device=True)


def test_repeated_calls_share_scratch(gpu, orc):
    rng = np.random.default_rng(6)
    for _ in range(5):
        check_dql(gpu, orc, rng.normal(0, rng.uniform(0.1, 10), size=70001).astype(np.float32),
                  device=True)


@pytest.mark.parametrize("signed", [False, True])
def test_quantize_linear(gpu, orc, signed):
    rng = np.random.default_rng(7)
    x = rng.normal(0, 40, size=(33, 129)).astype(np.float32)
    dt = np.int8 if signed else np.uint8
    zp = np.array(-3 if signed else 131, dt)
    want = orc.quantize(x, 0.37, float(zp), signed)
    got = gpu.quantize_linear(x, 0.37, zp, out_dtype=dt)
    assert np.array_equal(got, want)
    want = orc.quantize(x, 0.37, 0.0, signed)
    got = gpu.quantize_linear(x, 0.37, None, out_dtype=dt)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("scale", [2e-31, 1.1e-30, 3.3e-7, 0.1, 1 / 3, 0.99999994, 1.9999999, 255 / 7,
                                   8e29, 2e30, -0.3])
@pytest.mark.parametrize("zp,signed", [(0, False), (255, False), (77, False), (-128, True), (5, True)])
def test_quotients_next_to_ties(gpu, orc, scale, zp, signed):
    """Values whose quotient by the scale lies on a tie or a few ulps beside it, and
    values far beyond what saturates, for scales that take the divide-free
    arithmetic and for such that do not."""
    s = np.float32(scale)
    tie = ((np.arange(-300, 300) + 0.5).astype(np.float32) * s).astype(np.float32)
    near = [(tie.view(np.int32) + d).view(np.float32) for d in range(-3, 4)]
    far = np.array([0.0, -0.0, 1e-40, -1e-40, 1e38, -1e38, 3e38, -3e38, np.inf, -np.inf, np.nan],
                   np.float32)
    x = np.concatenate(near + [far, (np.arange(-300, 300) * s).astype(np.float32)])
    dt = np.int8 if signed else np.uint8
    got = gpu.quantize_linear(x, s, np.array(zp, dt), out_dtype=dt)
    want = orc.quantize(x, s, float(zp), signed)
    assert np.array_equal(got, want), (x[got != want][:8], got[got != want][:8], want[got != want][:8])


@pytest.mark.parametrize("dt", [np.uint8, np.int8, np.int32])
def test_dequantize_linear(gpu, orc, dt):
    rng = np.random.default_rng(8)
    info = np.iinfo(dt)
    x = rng.integers(max(info.min, -10**6), min(info.max, 10**6), size=(17, 65)).astype(dt)
    zp = np.array(5, dt)
    want = orc.dequantize_linear(x, 0.0123, 5)
    got = gpu.dequantize_linear(x, 0.0123, zp)
    assert got.tobytes() == want.tobytes()
    want = orc.dequantize_linear(x, 0.0123, 0)
    assert gpu.dequantize_linear(x, 0.0123, None).tobytes() == want.tobytes()


def test_argument_errors(gpu):
    with pytest.raises(gpu.OmcudaError) as ei:
        gpu.quantize_linear(np.ones((2, 3), np.float32), np.ones(3, np.float32))
    assert ei.value.code == gpu.ENOTSUP     # per-axis: rejected like the reference
    x = gpu.Tensor.from_numpy(np.ones(4, np.float32))
    y = gpu.Tensor.from_numpy(np.ones(5, np.uint8))
    s = gpu.Tensor.from_numpy(np.zeros((), np.float32))
    z = gpu.Tensor.from_numpy(np.zeros((), np.uint8))
    gpu.lib().omcudaDynamicQuantizeLinear(y.handle, s.handle, z.handle, x.handle)
    with pytest.raises(gpu.OmcudaError) as ei:
        gpu.check()
    assert ei.value.code == gpu.EINVAL


@pytest.mark.parametrize("n", [4, 4095, 8191, 8192, 8193, 65537, 131071, 131073, 262143, 262144,
                               262145])
def test_one_cluster_sizes(gpu, orc, n):
    # Up to 262144 values are reduced and quantized by one cluster that holds
    # them in registers: the sizes at which it grows, the last it takes and the
    # first it does not, on aligned data and on data that starts at an odd element
    # (and is written at an odd byte).
    import torch
    x = np.random.default_rng(n).normal(1, 3, size=n).astype(np.float32)
    check_dql(gpu, orc, x, device=True)
    xt = torch.zeros(n + 1, device="cuda")
    xt[1:] = torch.from_numpy(x).cuda()
    yt = torch.zeros(n + 2, dtype=torch.uint8, device="cuda")
    s, z = torch.zeros((), device="cuda"), torch.zeros((), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    t = [gpu.Tensor.from_cuda_array(a) for a in (yt[1:n + 1], s, z, xt[1:])]
    gpu.lib().omcudaDynamicQuantizeLinear(*[a.handle for a in t])
    gpu.check()
    torch.cuda.synchronize()
    want_y, want_s, want_z = orc.dynamic_quantize_linear(x)
    y = yt.cpu().numpy()
    assert np.array_equal(y[1:n + 1], want_y) and y[0] == 0 and y[n + 1] == 0
    assert s.item() == want_s and z.item() == want_z


@pytest.mark.parametrize("n", [3, 4096, 4099, 262147, 1048575, 9 << 20])
@pytest.mark.parametrize("shift", [0, 1])
def test_pass_run_edges(gpu, orc, n, shift):
    # QuantizeLinear and DequantizeLinear take runs of 4096 values per block: part
    # of a run, one whole run, one for each of many blocks (more than one per block:
    # test_pass_grid_wraps), and addresses that allow no vector access.
    import torch
    rng = np.random.default_rng(n)
    x = rng.normal(0, 20, size=n).astype(np.float32)
    xt = torch.zeros(n + 1, device="cuda")
    xt[shift:shift + n] = torch.from_numpy(x).cuda()
    qt = torch.zeros(n + 1, dtype=torch.uint8, device="cuda")
    q, xd = (gpu.Tensor.from_cuda_array(a[shift:shift + n]) for a in (qt, xt))
    zp = np.array(131, np.uint8)
    L = gpu.lib()
    s, z = gpu.Tensor.from_numpy(np.array(0.37, np.float32)), gpu.Tensor.from_numpy(zp)
    torch.cuda.synchronize()
    L.omcudaQuantizeLinear(q.handle, xd.handle, s.handle, z.handle)
    gpu.check()
    torch.cuda.synchronize()
    want = orc.quantize(x, 0.37, 131.0, False)
    got = qt.cpu().numpy()
    assert np.array_equal(got[shift:shift + n], want)
    assert not got[:shift].any() and not got[shift + n:].any()
    for dt in (np.uint8, np.int8, np.int32):
        src = torch.zeros(n + 1, dtype=getattr(torch, np.dtype(dt).name), device="cuda")
        vals = want.view(np.int8).astype(dt) if dt != np.uint8 else want
        src[shift:shift + n] = torch.from_numpy(vals).cuda()
        y = torch.full((n + 1,), -1.0, device="cuda")
        zpd = gpu.Tensor.from_numpy(np.array(5, dt))
        torch.cuda.synchronize()
        yd, sd = (gpu.Tensor.from_cuda_array(a[shift:shift + n]) for a in (y, src))
        L.omcudaDequantizeLinear(yd.handle, sd.handle, s.handle, zpd.handle)
        gpu.check()
        torch.cuda.synchronize()
        out = y.cpu().numpy()
        assert out[shift:shift + n].tobytes() == orc.dequantize_linear(vals, 0.37, 5).tobytes()
        assert (out[:shift] == -1).all() and (out[shift + n:] == -1).all()


@pytest.mark.parametrize("dt", [np.uint8, np.int8, np.int32])
@pytest.mark.parametrize("xs,ys", [(0, 0), (4, 4), (4, 1), (1, 4), (3, 2)])
@pytest.mark.parametrize("n", [1, 3, 5, 1023, 40001])
def test_dequantize_alignments(gpu, orc, dt, xs, ys, n):
    # Groups of four values where both tensors start on one, single values
    # where either does not; the last one to three values of a ragged size.
    import torch
    rng = np.random.default_rng(n)
    info = np.iinfo(dt)
    vals = rng.integers(max(info.min, -10**6), min(info.max, 10**6), size=n).astype(dt)
    src = torch.zeros(n + 8, dtype=getattr(torch, np.dtype(dt).name), device="cuda")
    src[xs:xs + n] = torch.from_numpy(vals).cuda()
    y = torch.full((n + 8,), -1.0, device="cuda")
    torch.cuda.synchronize()
    t = [gpu.Tensor.from_cuda_array(y[ys:ys + n]), gpu.Tensor.from_cuda_array(src[xs:xs + n]),
         gpu.Tensor.from_numpy(np.array(0.0123, np.float32))]
    for zp in (np.array(5, dt), None):
        z = gpu.Tensor.from_numpy(zp) if zp is not None else None
        gpu.lib().omcudaDequantizeLinear(*[a.handle for a in t], z.handle if z else None)
        gpu.check()
        torch.cuda.synchronize()
        out = y.cpu().numpy()
        want = orc.dequantize_linear(vals, 0.0123, 5 if zp is not None else 0)
        assert out[ys:ys + n].tobytes() == want.tobytes()
        assert (out[:ys] == -1).all() and (out[ys + n:] == -1).all()


@pytest.mark.parametrize("shift", [0, 1])
def test_pass_grid_wraps(gpu, orc, shift):
    # More values than one run of 4096 for each of the 64 blocks per SM a pass has at
    # most: some blocks take a second run, the last one a part of one.
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = sms * 64 * 4096 + 5 * 4096 + 1027
    rng = np.random.default_rng(36)
    x = rng.normal(0, 20, size=n).astype(np.float32)
    xt = torch.zeros(n + 1, device="cuda")
    xt[shift:shift + n] = torch.from_numpy(x).cuda()
    L = gpu.lib()
    xd = gpu.Tensor.from_cuda_array(xt[shift:shift + n])
    s = gpu.Tensor.from_numpy(np.array(0.37, np.float32))

    def out(dtype):
        buf = torch.zeros(n + 1, dtype=dtype, device="cuda")
        return buf, gpu.Tensor.from_cuda_array(buf[shift:shift + n])

    for dt, zp in ((torch.uint8, np.array(131, np.uint8)), (torch.int8, np.array(-3, np.int8))):
        q, qd = out(dt)
        z = gpu.Tensor.from_numpy(zp)
        torch.cuda.synchronize()
        L.omcudaQuantizeLinear(qd.handle, xd.handle, s.handle, z.handle)
        gpu.check()
        torch.cuda.synchronize()
        want = orc.quantize(x, 0.37, float(zp), dt == torch.int8)
        assert np.array_equal(q.cpu().numpy()[shift:shift + n], want)
        y, yd = out(torch.float32)
        torch.cuda.synchronize()
        L.omcudaDequantizeLinear(yd.handle, qd.handle, s.handle, z.handle)
        gpu.check()
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy()[shift:shift + n],
                              orc.dequantize_linear(want, 0.37, int(zp)))
    q, qd = out(torch.uint8)
    ys, yz = torch.zeros((), device="cuda"), torch.zeros((), dtype=torch.uint8, device="cuda")
    t = [gpu.Tensor.from_cuda_array(a) for a in (ys, yz)]
    torch.cuda.synchronize()
    L.omcudaDynamicQuantizeLinear(qd.handle, t[0].handle, t[1].handle, xd.handle)
    gpu.check()
    torch.cuda.synchronize()
    want_y, want_s, want_z = orc.dynamic_quantize_linear(x)
    assert np.array_equal(q.cpu().numpy()[shift:shift + n], want_y)
    assert ys.item() == want_s and yz.item() == want_z


@pytest.mark.parametrize("m,k", [(8, 1001), (9, 1001), (591, 1001), (592, 1001), (593, 1024), (591, 1024),
                                 (40, 8200), (5000, 67), (21, 4099),
                                 (1, 16381), (4, 4096), (16, 1009),
                                 (1, 70001), (3, 40000), (16, 4112), (17, 8192), (74, 4113), (75, 4113)])
@pytest.mark.parametrize("wt", [np.int8, np.uint8])
def test_quantized_rows(gpu, orc, m, k, wt):
    """The quantize pass by rows inside a linear, with (unsigned weights with a zero
    point) and without the rows' sums: one block's worth, several blocks, a block and a
    warp per row and the lines between them, rows that take wide loads and rows that do not."""
    rng = np.random.default_rng(m * 7 + k)
    x = rng.normal(0.3, 2, size=(m, k)).astype(np.float32)
    n = 33
    w = rng.integers(-127, 128, (k, n)).astype(np.int8) if wt == np.int8 else \
        rng.integers(0, 256, (k, n)).astype(np.uint8)
    zp = None if wt == np.int8 else np.array(131, np.uint8)
    bias = rng.normal(size=n).astype(np.float32)
    xq, xs, xz = orc.dynamic_quantize_linear(x)
    wi = w.astype(np.int64) - (0 if zp is None else 131)
    acc = (xq.astype(np.int64) - int(xz)) @ wi
    want = (acc.astype(np.float32) * np.float32(np.float32(xs) * np.float32(0.0157))) + bias
    got = gpu.dyn_quant_linear(x, w, np.float32(0.0157), zp, bias, 0)
    assert got.tobytes() == want.astype(np.float32).tobytes()


@pytest.mark.parametrize("n", [65537, 100001, 262144])
def test_captured_dynamic_quantize_needs_no_pool(gpu, orc, n):
    """Above the size that is fastest in one launch a captured call stays one all the
    same: two passes would leave their partials in a pool block, which the replays
    would write to after it was given back."""
    import torch
    rng = np.random.default_rng(n)
    x = torch.empty(n, device="cuda")
    y = torch.zeros(n, dtype=torch.uint8, device="cuda")
    s, z = torch.zeros((), device="cuda"), torch.zeros((), dtype=torch.uint8, device="cuda")
    call = [gpu.Tensor.from_cuda_array(t) for t in (y, s, z, x)]
    L = gpu.lib()
    gpu.dynamic_quantize_linear(np.ones(n, np.float32))  # (kernels loaded, a free pool block)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    try:
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            L.omcudaSetStream(stream.cuda_stream)
            before = gpu.launch_count()
            L.omcudaDynamicQuantizeLinear(*[t.handle for t in call])
            launches = gpu.launch_count() - before
    finally:
        L.omcudaSetStream(None)
    gpu.check()
    assert launches == 1
    for _ in range(2):
        v = rng.normal(0.1, 3, size=n).astype(np.float32)
        x.copy_(torch.from_numpy(v))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        want_y, want_s, want_z = orc.dynamic_quantize_linear(v)
        assert np.array_equal(y.cpu().numpy(), want_y)
        assert s.item() == want_s and z.item() == want_z


@pytest.mark.parametrize("n", [1000, 65537, 131072, 262144])
@pytest.mark.parametrize("where", ["y", "y_end", "scalars"])
def test_dynamic_quantize_onto_its_input(gpu, orc, n, where):
    """Outputs in the memory of x, for sizes that one cluster holds."""
    import torch
    v = np.random.default_rng(n).normal(-0.2, 3, size=n).astype(np.float32)
    xt = torch.from_numpy(v).cuda()
    raw = xt.view(torch.uint8)
    y = {"y": raw[:n], "y_end": raw[3 * n:], "scalars": torch.zeros(n, dtype=torch.uint8, device="cuda")}[where]
    s, z = torch.zeros(1, device="cuda"), torch.zeros(1, dtype=torch.uint8, device="cuda")
    if where == "scalars":
        s, z = xt[n - 1:], raw[:1]
    t = [gpu.Tensor.from_cuda_array(a) for a in (y, s, z, xt)]
    torch.cuda.synchronize()
    gpu.lib().omcudaDynamicQuantizeLinear(*[a.handle for a in t])
    gpu.synchronize()
    torch.cuda.synchronize()
    want_y, want_s, want_z = orc.dynamic_quantize_linear(v)
    assert np.array_equal(y.cpu().numpy(), want_y)
    assert s.item() == want_s and z.item() == want_z


@pytest.mark.parametrize("n", [1, 3, 255, 1025, 70001, 1300001])
@pytest.mark.parametrize("xs,ys", [(1, 0), (2, 1), (3, 3), (0, 1), (0, 2), (0, 4)])
def test_quantize_alignments(gpu, orc, n, xs, ys):
    """Tensors that start anywhere, with scales that take the divide-free arithmetic
    and one that does not; nothing beside the result is written."""
    import torch
    rng = np.random.default_rng(n + xs + 4 * ys)
    v = rng.normal(0, 20, size=n).astype(np.float32)
    xt = torch.zeros(n + 4, device="cuda")
    xt[xs:xs + n] = torch.from_numpy(v).cuda()
    xd = gpu.Tensor.from_cuda_array(xt[xs:xs + n])
    L = gpu.lib()

    def result(dtype):
        buf = torch.full((n + 16,), 99, dtype=dtype, device="cuda")
        return buf, gpu.Tensor.from_cuda_array(buf[ys:ys + n])

    def check(buf, want):
        got = buf.cpu().numpy()
        assert np.array_equal(got[ys:ys + n], want)
        assert (got[:ys] == 99).all() and (got[ys + n:] == 99).all()

    for scale, zp in ((0.37, np.array(131, np.uint8)), (0.21, np.array(-3, np.int8)),
                      (1e-33, np.array(7, np.uint8))):
        buf, yd = result(getattr(torch, zp.dtype.name))
        s, z = gpu.Tensor.from_numpy(np.array(scale, np.float32)), gpu.Tensor.from_numpy(zp)
        torch.cuda.synchronize()
        L.omcudaQuantizeLinear(yd.handle, xd.handle, s.handle, z.handle)
        gpu.synchronize()
        check(buf, orc.quantize(v, scale, float(zp), zp.dtype == np.int8))
    buf, yd = result(torch.uint8)
    s, z = torch.zeros((), device="cuda"), torch.zeros((), dtype=torch.uint8, device="cuda")
    t = [gpu.Tensor.from_cuda_array(a) for a in (s, z)]
    torch.cuda.synchronize()
    L.omcudaDynamicQuantizeLinear(yd.handle, t[0].handle, t[1].handle, xd.handle)
    gpu.synchronize()
    want_y, want_s, want_z = orc.dynamic_quantize_linear(v)
    check(buf, want_y)
    assert s.item() == want_s and z.item() == want_z


@pytest.mark.parametrize("n", [113700, 802815, 802821, 2424830, 2424833, 4849663, 4849668, 9699333])
@pytest.mark.parametrize("at", [0.0, 0.37, 1.0])
def test_dynamic_quantize_extremes_of_deep_and_full_blocks(gpu, orc, n, at):
    """The reduction's forms (runs of one to eight groups; up to one, one to two and more
    blocks of 16384 values per SM; single values): an extreme anywhere is found."""
    x = np.random.default_rng(n).normal(size=4096).astype(np.float32)
    x = np.resize(x, n)
    i = min(int(at * n), n - 2)
    x[i], x[i + 1] = 77.0, -55.0
    check_dql(gpu, orc, x, device=True)


@pytest.mark.parametrize("n", [200000, 262147, 4000003])
def test_wide_pass_of_zeros(gpu, orc, n):
    x = np.zeros(n, np.float32)
    x[::3] = -0.0
    check_dql(gpu, orc, x, device=True)
    x[5::7] = np.nan
    with np.errstate(all="ignore"):
        check_dql(gpu, orc, x, device=True)


# Ranges whose 255th part is no longer a positive fp32 number although not all values are zero
# (127 steps of the least denormal and fewer), the first ranges above, denormal and least scales.
TINY = {"positive": (1e-44, 2e-44, 1e-43, 0.0, -0.0), "both": (1e-44, -2e-44, 1e-43, 0.0),
        "least": (1.4e-45, 0.0, 0.0), "negative": (-7e-44, 0.0, np.nan),
        "mostly zeros": (0.0,) * 4099 + (7e-44,), "step of scale": (1.79e-43, 0.0, 1e-44),
        "denormal scale": (1e-40, -3e-39, 0.0), "least normal": (1.2e-38, -2.3e-38, 1e-44)}


@pytest.mark.parametrize("n", [199999, 200000, 4000003])
@pytest.mark.parametrize("xs", [0, 4])
@pytest.mark.parametrize("values", sorted(TINY))
def test_wide_pass_of_denormals(gpu, orc, n, xs, values):
    import torch
    v = np.resize(np.array(TINY[values], np.float32), n)
    xt = torch.zeros(n + 4, device="cuda")
    xt[xs:xs + n] = torch.from_numpy(v).cuda()
    y = torch.full((n + 8,), 99, dtype=torch.uint8, device="cuda")
    s, z = torch.zeros((), device="cuda"), torch.zeros((), dtype=torch.uint8, device="cuda")
    t = [gpu.Tensor.from_cuda_array(a) for a in (y[:n], s, z, xt[xs:xs + n])]
    torch.cuda.synchronize()
    gpu.lib().omcudaDynamicQuantizeLinear(*[a.handle for a in t])
    gpu.synchronize()
    with np.errstate(all="ignore"):
        want_y, want_s, want_z = orc.dynamic_quantize_linear(v)
    assert s.cpu().numpy().tobytes() == want_s.tobytes() and z.item() == want_z
    got = y.cpu().numpy()
    assert np.array_equal(got[:n], want_y) and (got[n:] == 99).all()


@pytest.mark.parametrize("n", [200000, 212999])
@pytest.mark.parametrize("scale", [1.4e-45, 7e-45, 5e-40, 1.1754944e-38, 9.9e-31, 1e-30, 1.0000001e-30,
                                   0.99e30, 1e30, 3e32, 1.3e38, 3.4e38, np.inf, np.nan, -0.0, -0.5, -1e-40])
def test_wide_pass_of_scales_that_are_not_ordinary(gpu, orc, n, scale):
    """Ties, their neighbours and all that saturates, under scales whose reciprocal or
    residuals fp32 does not hold (those between are divided by with multiplications alone)."""
    import torch
    rng = np.random.default_rng(n)
    s = np.float32(scale)
    with np.errstate(all="ignore"):
        k = rng.integers(-600, 600, size=n) * 0.5 + rng.choice([0.0, 1e-6, -1e-6, 0.2], size=n)
        v = (k * (np.float64(s) if np.isfinite(s) else 1.0)).astype(np.float32)
    v[::3] = np.nextafter(v[::3], np.float32(0))
    v[1::501] = rng.normal(0, 1, size=v[1::501].size)
    v[:8] = (np.inf, -np.inf, np.nan, 3.4e38, -3.4e38, 1.4e-45, -1.4e-45, -0.0)
    v[-3:] = v[2:5]
    x, st = torch.from_numpy(v).cuda(), torch.tensor(scale, device="cuda")
    for zp in (np.array(131, np.uint8), np.array(-7, np.int8), np.array(0, np.uint8)):
        y, z = torch.empty(n, dtype=getattr(torch, zp.dtype.name), device="cuda"), torch.tensor(zp).cuda()
        t = [gpu.Tensor.from_cuda_array(a) for a in (y, x, st, z)]
        torch.cuda.synchronize()
        gpu.lib().omcudaQuantizeLinear(*[a.handle for a in t])
        gpu.synchronize()
        with np.errstate(all="ignore"):
            want = orc.quantize(v, s, float(zp), zp.dtype == np.int8)
        assert np.array_equal(y.cpu().numpy(), want)


@pytest.mark.parametrize("n", [199999, 200000, 212999])
@pytest.mark.parametrize("flags", [0, 2])  # 2: OMCUDA_MODE_FAST_MATH, x times the rounded reciprocal
@pytest.mark.parametrize("scale", [1.4e-45, 3e-39, 1e-32, 0.05, 3e32, 3.4e38, np.inf, np.nan])
def test_wide_pass_of_scales_of_either_sign_in_both_modes(gpu, orc, n, flags, scale):
    import torch
    rng = np.random.default_rng(n + flags)
    for s in (np.float32(scale), -np.float32(scale)):
        with np.errstate(all="ignore"):
            k = rng.integers(-600, 600, size=n) * 0.5 + rng.choice([0.0, 1e-6, -1e-6, 0.2], size=n)
            v = (k * (np.float64(s) if np.isfinite(s) else 1.0)).astype(np.float32)
        v[::3] = np.nextafter(v[::3], np.float32(0))
        v[1::501] = rng.normal(0, 1, size=v[1::501].size)
        v[:8] = (np.inf, -np.inf, np.nan, 3.4e38, -3.4e38, 1.4e-45, -1.4e-45, -0.0)
        v[-3:] = v[:3]
        x, st = torch.from_numpy(v).cuda(), torch.tensor(float(s), device="cuda")
        for zp in (np.array(131, np.uint8), np.array(-7, np.int8)):
            y, z = torch.empty(n, dtype=getattr(torch, zp.dtype.name), device="cuda"), torch.tensor(zp).cuda()
            t = [gpu.Tensor.from_cuda_array(a) for a in (y, x, st, z)]
            torch.cuda.synchronize()
            try:
                gpu.lib().omcudaSetQuantizationMode(flags)
                gpu.lib().omcudaQuantizeLinear(*[a.handle for a in t])
                gpu.synchronize()
            finally:
                gpu.lib().omcudaSetQuantizationMode(0)
            with np.errstate(all="ignore"):
                if flags:
                    q = np.rint(v * (np.float32(1) / s)) + np.float32(zp)
                    lim = np.iinfo(zp.dtype)
                    want = np.fmin(np.fmax(q, np.float32(lim.min)), np.float32(lim.max)).astype(zp.dtype)
                else:
                    want = orc.quantize(v, s, float(zp), zp.dtype == np.int8)
            assert np.array_equal(y.cpu().numpy(), want)


# (from 606209 values the blocks are two per SM, from 1212417 three, then four)
@pytest.mark.parametrize("n", [23999, 24000, 24007, 606208, 606209, 700001, 1212417, 1500003, 2000000])
@pytest.mark.parametrize("values", ["normal", "zeros", "no range"] + sorted(TINY))
def test_quantize_from_range(gpu, orc, n, values):
    """What an encoder's linears do to a tensor whose range its producer has kept.  "no range":
    a range of nothing but zero beside values that are not; they are quantized with it."""
    import ctypes

    import torch
    rng = np.random.default_rng(n)
    v = np.resize(np.zeros(1, np.float32) if values == "zeros" else
                  np.array(TINY[values], np.float32) if values in TINY else
                  rng.normal(0, 3, size=65537).astype(np.float32), n)
    of = np.zeros(1, np.float32) if values == "no range" else v
    x, f = torch.from_numpy(v).cuda(), torch.from_numpy(of).cuda()
    y = torch.full((n + 8,), 99, dtype=torch.uint8, device="cuda")
    par = torch.zeros(4, device="cuda")
    ranges = torch.zeros(2, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    L, st = gpu.lib(), ctypes.c_void_p(gpu.lib().omcudaGetStream())
    from omcuda import dev
    dev.range_init(ranges.data_ptr(), 1, st)
    assert L.omcudaDevRangeFold(ctypes.c_void_p(f.data_ptr()), ctypes.c_int64(of.size),
                                ctypes.c_void_p(ranges.data_ptr()), st) == 0
    dev.quantize_from_range(x.data_ptr(), n, ranges.data_ptr(), y.data_ptr(), par.data_ptr(),
                            par.data_ptr() + 8, par.data_ptr() + 12, st)
    gpu.synchronize()
    with np.errstate(all="ignore"):
        want_y, want_s, want_z = orc.dynamic_quantize_linear(of)
        if values == "no range":
            want_y = orc.quantize(v, want_s, float(want_z), False)
    p, got = par.cpu().numpy(), y.cpu().numpy()
    assert p[0].tobytes() == want_s.tobytes() == p[2].tobytes() and p[1] == want_z
    assert p[3:].view(np.uint8)[0] == want_z
    assert np.array_equal(got[:n], want_y) and (got[n:] == 99).all()


@pytest.mark.parametrize("n", [199999, 200000, 200007, 204800, 204801, 208897, 3031041, 39010313])
@pytest.mark.parametrize("xs,ys", [(0, 0), (8, 8), (4, 0), (0, 4)])
def test_wide_pass(gpu, orc, n, xs, ys):
    """The pass with 32-byte loads: from 200000 values, where x starts on 32 bytes and y on 8
    (else the 16-byte one), runs of 4096, what is left of them, more runs than resident
    blocks; a scale it takes, scales left to the divide, and DynamicQuantizeLinear."""
    import torch
    rng = np.random.default_rng(n)
    v = np.resize(rng.normal(0, 20, size=65537).astype(np.float32), n)
    v[-3:] = (np.inf, -1e30, np.nan)
    xt = torch.zeros(n + 8, device="cuda")
    xt[xs:xs + n] = torch.from_numpy(v).cuda()
    xd = gpu.Tensor.from_cuda_array(xt[xs:xs + n])
    L = gpu.lib()
    buf = torch.empty(n + 16, dtype=torch.uint8, device="cuda")

    def check(want):
        got = buf.cpu().numpy()
        assert np.array_equal(got[ys:ys + n], want.view(np.uint8))
        assert (got[:ys] == 99).all() and (got[ys + n:] == 99).all()

    for scale, zp in ((0.37, np.array(131, np.uint8)), (0.21, np.array(-3, np.int8)),
                      (0.0, np.array(7, np.uint8)), (1e-33, np.array(-7, np.int8))):
        buf.fill_(99)
        yt = buf[ys:ys + n] if zp.dtype == np.uint8 else buf.view(torch.int8)[ys:ys + n]
        s, z = gpu.Tensor.from_numpy(np.array(scale, np.float32)), gpu.Tensor.from_numpy(zp)
        torch.cuda.synchronize()
        yd = gpu.Tensor.from_cuda_array(yt)
        L.omcudaQuantizeLinear(yd.handle, xd.handle, s.handle, z.handle)
        gpu.synchronize()
        with np.errstate(all="ignore"):
            check(orc.quantize(v, scale, float(zp), zp.dtype == np.int8))
    v[-3:] = 0
    xt[xs + n - 3:xs + n] = 0
    buf.fill_(99)
    s, z = torch.zeros((), device="cuda"), torch.zeros((), dtype=torch.uint8, device="cuda")
    t = [gpu.Tensor.from_cuda_array(a) for a in (s, z, buf[ys:ys + n])]
    torch.cuda.synchronize()
    L.omcudaDynamicQuantizeLinear(t[2].handle, t[0].handle, t[1].handle, xd.handle)
    gpu.synchronize()
    want_y, want_s, want_z = orc.dynamic_quantize_linear(v)
    check(want_y)
    assert s.item() == want_s and z.item() == want_z


@pytest.mark.parametrize("n", [65541, 75775, 113663, 113664, 113665, 114177])
@pytest.mark.parametrize("at", ["first", "middle", "last"])
def test_dynamic_quantize_extremes_of_small_blocks(gpu, orc, n, at):
    # Around the line (1.5 blocks of 512 values per SM) where the reduction changes its
    # blocks, with the one value that decides the scale where a block could miss it.
    x = np.random.default_rng(n).normal(size=n).astype(np.float32)
    x[{"first": 0, "middle": n // 2, "last": n - 1}[at]] = -40.0
    y, s, z = gpu.dynamic_quantize_linear(x, device=False)
    ry, rs, rz = orc.dynamic_quantize_linear(x)
    assert s == rs and z == rz and np.array_equal(y, ry)
