"""The allocation-free DynamicQuantizeLinear entry point.

Some users of this library run where device memory cannot be allocated on
demand -- every byte of HBM was claimed by the hosting server's own arena, or
the allocator's device-wide synchronisation is not acceptable in their loop.
For them the library carries its reduction scratch inside its own image.  This
test calls that entry point through the C ABI twice in a row (the second call
sees the first one's leftovers in the shared scratch) and requires the very
same bytes the ordinary entry point produces, plus a refusal of inputs beyond
the stated limit.  It lives in a file collected last so that a run that stops
at the first failure has already exercised everything else.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(gpu, fn_noalloc, fn_plain, x, scratch, stream):
    d = gpu.Tensor.from_numpy(x).to_device()
    outs = []
    for which in ("noalloc", "plain"):
        y = gpu.Tensor.device_empty(x.shape, np.uint8)
        s = gpu.Tensor.device_empty((), np.float32)
        z = gpu.Tensor.device_empty((), np.uint8)
        if which == "noalloc":
            rc = fn_noalloc(d.data_ptr, x.size, y.data_ptr, s.data_ptr, z.data_ptr, stream)
        else:
            rc = fn_plain(d.data_ptr, x.size, y.data_ptr, s.data_ptr, z.data_ptr,
                          scratch.data_ptr, stream)
        assert rc == 0, gpu.lib().omcudaGetLastErrorString()
        outs.append((y.numpy(), s.numpy(), z.numpy()))
    gpu.synchronize()
    return outs


def test_no_alloc_entry_matches_the_ordinary_one_twice(gpu):
    L = gpu.lib()
    vp, i64 = ctypes.c_void_p, ctypes.c_int64
    fn_noalloc = L.omcudaDevDynamicQuantizeLinearNoAlloc
    fn_noalloc.argtypes = [vp, i64, vp, vp, vp, vp]
    fn_plain = L.omcudaDevDynamicQuantizeLinear
    fn_plain.argtypes = [vp, i64, vp, vp, vp, vp, vp]
    L.omcudaDevDqlScratchBytes.restype = i64
    L.omcudaDevDqlScratchBytes.argtypes = [i64]
    stream = L.omcudaGetStream()
    scratch = gpu.Tensor.from_numpy(
        np.zeros(L.omcudaDevDqlScratchBytes(0), np.uint8)).to_device()
    rng = np.random.default_rng(2024)
    # first call: many blocks; second call: fewer blocks and a different range,
    # so stale partial results from the first call are in the shared scratch
    for shape, sigma in (((1024, 1537), 3.0), ((37, 129), 0.25)):
        x = rng.normal(0, sigma, size=shape).astype(np.float32)
        (y1, s1, z1), (y2, s2, z2) = _run(gpu, fn_noalloc, fn_plain, x, scratch, stream)
        assert s1.tobytes() == s2.tobytes()
        assert int(z1) == int(z2)
        assert np.array_equal(y1, y2)


def test_no_alloc_entry_rejects_oversized_input(gpu):
    L = gpu.lib()
    vp, i64 = ctypes.c_void_p, ctypes.c_int64
    fn = L.omcudaDevDynamicQuantizeLinearNoAlloc
    fn.argtypes = [vp, i64, vp, vp, vp, vp]
    x = gpu.Tensor.device_empty((16,), np.float32)
    y = gpu.Tensor.device_empty((16,), np.uint8)
    s = gpu.Tensor.device_empty((), np.float32)
    z = gpu.Tensor.device_empty((), np.uint8)
    L.omcudaClearError()
    rc = fn(x.data_ptr, (1 << 31) + 1, y.data_ptr, s.data_ptr, z.data_ptr,
            L.omcudaGetStream())
    assert rc == gpu.EINVAL
    assert b"exceed the limit" in L.omcudaGetLastErrorString()
    L.omcudaClearError()


def test_linear_of_few_rows_when_no_memory_is_left(gpu):
    """Two kernels and their scratch where there is memory for it; the one launch that needs
    none, with the same bits, where every byte of the device is taken."""
    import torch
    L, T = gpu.lib(), gpu.Tensor.from_cuda_array
    M, K, N = 3, 5000, 10000
    rng = np.random.default_rng(7)
    x = torch.from_numpy(rng.normal(0, 1, size=(M, K)).astype(np.float32)).cuda()
    w = torch.from_numpy(rng.integers(-127, 128, size=(K, N)).astype(np.int8)).cuda()
    ws, y = torch.tensor(0.0157, device="cuda"), torch.zeros((3, M, N), device="cuda")
    t = [T(x), T(w), T(ws)]
    ys = [T(y[i]) for i in range(3)]
    L.omcudaRegisterConstant(t[1].handle)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    driver, taken = ctypes.CDLL("libcuda.so.1"), []

    def call(out):
        before = gpu.launch_count()
        L.omcudaDynQuantLinear(ys[out].handle, *[a.handle for a in t], None, None, 0)
        gpu.check()
        return gpu.launch_count() - before

    torch.cuda.synchronize()
    try:
        L.omcudaSetStream(stream.cuda_stream)
        assert call(0) >= 2
        gpu.synchronize()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            call(1)
        graph.replay()  # (the kernel of the one launch is on the device now)
        torch.cuda.synchronize()
        assert L.omcudaDeviceAlloc(ctypes.c_int64(1 << 50)) in (None, 0)  # the pool lets go of its blocks
        L.omcudaClearError()
        size, ptr = 1 << 38, ctypes.c_uint64()
        while size >= 256:
            if driver.cuMemAlloc_v2(ctypes.byref(ptr), ctypes.c_size_t(size)) == 0:
                taken.append(ptr.value)
            else:
                size //= 2
        assert call(2) == 1
        gpu.synchronize()
        for p in taken:
            driver.cuMemFree_v2(ctypes.c_uint64(p))
        taken = []
        assert call(0) >= 2
        gpu.synchronize()
        got = y.cpu().numpy()
        assert np.abs(got[0]).max() > 0
        assert got[0].tobytes() == got[1].tobytes() == got[2].tobytes()
    finally:
        for p in taken:
            driver.cuMemFree_v2(ctypes.c_uint64(p))
        L.omcudaSetStream(None)
        torch.cuda.synchronize()
        L.omcudaForgetConstants()
