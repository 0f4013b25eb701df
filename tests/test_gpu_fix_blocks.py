"""The exact recomputation of Q/K/V sign bits by blocks of 32 steps, against the oracle bit for bit: widths at the edges of its
warps and chunks, blocks that end inside 32 steps, from few flagged outputs to all of them (many times the queue), in an odd
part of the rows; exact sums of 0 and of -0.  With few blocks a CTA has 4 steps of one."""
import numpy as np
import pytest

from test_gpu_ops import _rosa_params, unpack_plane
from ullis_b200 import cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,d", [(1, 33, 64), (2, 31, 192), (3, 70, 256), (1, 65, 320), (2, 96, 512), (2, 37, 1024), (1, 40, 1088),
                                   (80, 70, 128), (151, 33, 64), (700, 31, 64)])   # parts of 8 and 16 steps, whole blocks
@pytest.mark.parametrize("small", ["none", "some", "all"])
def test_flagged_signs_are_those_of_the_oracle(oracle, B, T, d, small):
    rng = np.random.default_rng([B * T + d, len(small)])
    p = _rosa_params(rng, d)
    x = rng.standard_normal((B * T, d)).astype(np.float32)
    if small != "none":                               # sums below the absolute part of the error band: every output is flagged
        rows = rng.random(B * T) < (0.3 if small == "some" else 2.0)
        x[rows] *= np.float32(1e-8)
        x[rows, ::7] = np.float32(-0.0)
        x[0] = 0.0
        x[-1] = np.float32(-0.0)
        for m in "qkv":
            p[m]["bias"] = np.zeros(d, np.uint16)
    rt = cuda.CudaRuntime(0)
    try:
        got = rt.rosa_block_forward(x.ravel(), p, B, T, d)
        rt.kernel_timing(True)
        rt.rosa_block_forward(x.ravel(), p, B, T, d)
        assert ("fix_block" if d <= 1024 else "sign_fixup") in rt.kernel_times()
        rt.kernel_timing(False)
    finally:
        rt.close()
    _, want = oracle.rosa_block_forward(x.ravel(), p, B, T, d, taps=True)
    for m in "qkv":
        assert np.array_equal(unpack_plane(got[m + "_plane"], B * T * d), want[m + "_bits"]), m
    assert np.array_equal(got["idx"], want["idx"])


@pytest.mark.parametrize("name", ["ULLIS_CUDA_FIX_BLOCKS", "ULLIS_CUDA_FIX_LIST"])
def test_the_switch_by_either_name(monkeypatch, name):
    monkeypatch.setenv(name, "0")
    rt = cuda.CudaRuntime(0)
    try:
        x = np.random.default_rng(3).standard_normal((66, 64)).astype(np.float32)
        rt.kernel_timing(True)
        rt.rosa_block_forward(x.ravel(), _rosa_params(np.random.default_rng(4), 64), 2, 33, 64)
        ran = rt.kernel_times()
        assert "sign_fixup" in ran and "fix_block" not in ran
    finally:
        rt.close()
