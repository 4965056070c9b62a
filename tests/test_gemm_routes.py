"""Which products the kernel for few rows takes, and that the switches which name a tile
width, epilogue warps or a number of slices of the other tensor-core kernels reach those."""
import os
import random
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "onnx-mlir_b200")
SWITCHES = ("OMCUDA_GEMM_BN", "OMCUDA_GEMM_EW", "OMCUDA_GEMM_SPLIT_K", "OMCUDA_GEMV",
            "OMCUDA_GEMV_MMA_MAX_M")


def child(code, **switches):
    """The output of a process of its own: switches are read once."""
    env = {k: v for k, v in os.environ.items() if k not in SWITCHES}
    env.update(switches, PYTHONPATH=PKG)
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout.split()


@pytest.mark.parametrize("switches,taken", [
    ({}, (True, True, True, True)), ({"OMCUDA_GEMM_SPLIT_K": "0"}, (True, True, True, True)),
    ({"OMCUDA_GEMM_SPLIT_K": "3"}, (True, False, False, False)),
    ({"OMCUDA_GEMM_BN": "128"}, (True, False, False, False)),
    ({"OMCUDA_GEMM_BN": "512"}, (True, False, False, False)),
    ({"OMCUDA_GEMM_EW": "8"}, (True, False, False, False)),
    ({"OMCUDA_GEMM_EW": "16", "OMCUDA_GEMV": "0"}, (False, False, False, False))])
def test_switches_of_the_large_tiles_reach_them(built, switches, taken):
    # 16 rows are the GEMV kernels' without the few-rows kernel, unless those are off
    out = child("from omcuda import dev\n"
                "for s in ((16, 4096, 14336), (17, 768, 768), (64, 768, 768), (256, 768, 768)):\n"
                "    print(dev.gemm_few_plan(*s) is not None)", **switches)
    assert out == [str(t) for t in taken]


@pytest.mark.gpu
def test_forced_slices_are_launched(built):
    # 64 x 1024 x 512 in two slices: the pass over them, and the one that adds them up.
    code = """
import sys
import numpy as np
sys.path.insert(0, %r)
import omcuda
from omcuda import dev
from gpu_util import DevGemm
omcuda.init()
rng = np.random.default_rng(0)
A = rng.integers(0, 256, (64, 1024), dtype=np.uint8)
B = rng.integers(-128, 128, (1024, 512), dtype=np.int8)
dg = DevGemm(omcuda)
pb, keep = dg.prepare(B)
dA, Y = dg.dtensor(A), omcuda.Tensor.device_empty((64, 512), np.int32)
g = dev.GemmArgs()
g.M, g.N, g.K, g.A, g.a_signed, g.B = 64, 512, 1024, dA.data_ptr, 0, pb
g.epilogue, g.Y = dev.EPI_I32, Y.data_ptr
before = omcuda.launch_count()
dev.gemm_i8(g, dg.stream)
print(omcuda.launch_count() - before,
      np.array_equal(Y.numpy(), A.astype(np.int64) @ B.astype(np.int64)))
""" % os.path.join(ROOT, "tests")
    assert child(code, OMCUDA_GEMM_SPLIT_K="2") == ["2", "True"]
    assert child(code) == ["1", "True"]


def cheapest_cut(M, N, K, sms=148):
    """The cut with the least estimate (whole ceilings, no shortcuts)."""
    ceil = lambda a, b: -(-a // b)
    kb, best = ceil(K, 128), None
    for t in (16, 32, 64, 128):
        if t > 16 and t >= 2 * M:
            break
        for split in (1, 2, 3, 4, 6, 8):
            if split > kb:
                break
            ctas, kbs = ceil(N, 128) * ceil(M, t) * split, ceil(kb, split)
            found = sms * (3 if split > 2 else 4) // 4 - (8 if split == 2 else 0)
            steps = ceil(kbs, 2)
            besides = 2048 + (split * ceil(t, split) * 512 if split > 1 else 0)
            for stages in range(min(steps, 6), 0, -1):
                smem = max(stages * 256 * (128 + t), t * 512) + besides
                if smem <= 226 << 10 and smem * min(ceil(ctas, found), 3) <= 228 << 10:
                    break
            if smem > 226 << 10:
                continue
            rounds = ceil(ctas, found * min((228 << 10) // smem, 3))
            per_sm = float(ceil(ceil(ctas, rounds), sms))
            us = rounds * (max(per_sm * kbs * (16.0 + t / 8.0) * 0.0014, per_sm * kbs * 0.07,
                               steps * 0.109 * (1.0 + 3.86 / stages)) +
                           per_sm * min(t, M) * 0.0229) + ctas * 0.0037
            if best is None or us < best[0]:
                best = (us, t, split)
    return best[1:]


def test_the_plan_is_the_cheapest_cut(omcuda):
    from omcuda import dev
    rng, seen = random.Random(3), set()
    for _ in range(6000):
        M = rng.choice((rng.randint(2, 64), rng.randint(2, 640)))
        K, N = rng.randint(1, rng.choice((600, 16384))), rng.randint(1, rng.choice((600, 16384, 1 << 20)))
        plan = dev.gemm_few_plan(M, N, K)
        if plan is not None:
            seen.add(plan)
            assert plan == cheapest_cut(M, N, K), (M, N, K)
    assert len(seen) > 20
