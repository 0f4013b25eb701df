"""The results of a ROSA block: sign planes of whole and broken blocks of steps and of channel counts that are not whole words, into
page-locked memory by a kernel (small) or by copies (large), and into ordinary arrays."""
import ctypes as C

import numpy as np
import pytest

from conftest import unpack_plane
from ullis_b200 import cuda

pytestmark = pytest.mark.gpu


def f16(x):
    return np.asarray(x, np.float32).astype(np.float16).view(np.uint16)


def params(rng, d):
    p = {m: f16(rng.uniform(0, 1, d)) for m in ("x_q", "x_k", "x_v")}
    for m in "qkvo":
        p[m] = {"bits": rng.integers(0, 2 ** 32, (d * d + 31) // 32, dtype=np.uint32), "scale": f16(rng.uniform(0.005, 0.02, d)),
                "bias": f16(rng.normal(0, 0.01, d))}
        if d * d % 32:
            p[m]["bits"][-1] &= np.uint32((1 << d * d % 32) - 1)
    p["e"] = f16(rng.normal(0, 0.02, d))
    return p


@pytest.mark.parametrize("ordinary", [False, True])
@pytest.mark.parametrize("B,T,d", [(1, 1, 64), (2, 33, 64), (3, 300, 96), (1, 65, 40), (2, 31, 36), (1, 513, 64), (2, 700, 576)])
def test_planes_idx_and_outputs(cuda_rt, oracle, monkeypatch, B, T, d, ordinary):
    if ordinary:
        monkeypatch.setattr(cuda.CudaRuntime, "_empty", lambda self, shape, dtype: np.empty(shape, dtype))
    rng = np.random.default_rng([B, T, d])
    p, x, n = params(rng, d), rng.standard_normal(B * T * d).astype(np.float32), B * T * d
    ref, t = oracle.rosa_block_forward(x, p, B, T, d, taps=True)
    cuda_rt.set_mode(cuda.MODE_EXACT)
    try:
        got = cuda_rt.rosa_block_forward(x, p, B, T, d)
    finally:
        cuda_rt.set_mode(cuda.MODE_FAST)
    for m in "qkv":
        assert np.array_equal(unpack_plane(got[m + "_plane"], n), t[m + "_bits"]), m
    assert np.array_equal(got["idx"], t["idx"]) and np.array_equal(got["y"], t["y"]) and np.array_equal(got["out"], ref)


def test_a_block_that_was_freed_is_no_longer_written_by_kernels(cuda_rt):
    """The memory of a freed block may come back as ordinary memory: the call has to take the copy engine then."""
    rng = np.random.default_rng(5)
    d, T = 64, 32
    p, x = params(rng, d), rng.standard_normal(T * d).astype(np.float32)
    want = cuda_rt.rosa_block_forward(x, p, 1, T, d)
    block = C.c_void_p()
    cuda_rt._check(cuda_rt._lib.ullis_cuda_host_alloc(cuda_rt._h, C.c_size_t(1 << 16), C.byref(block)))
    cuda_rt._lib.ullis_cuda_host_free(block)
    keep = [np.empty(1 << 16, np.uint8) for _ in range(64)]
    cuda_rt.kernel_timing(True)
    original = cuda.CudaRuntime._empty
    try:
        cuda.CudaRuntime._empty = lambda self, shape, dtype: np.empty(shape, dtype)
        got = cuda_rt.rosa_block_forward(x, p, 1, T, d)
        ran = cuda_rt.kernel_times()
    finally:
        cuda.CudaRuntime._empty = original
        cuda_rt.kernel_timing(False)
    assert "copies_to_host" not in ran and len(keep) == 64
    assert all(np.array_equal(got[k], want[k]) for k in want)
