"""Sequence lengths that are no multiple of 32 through the tensor-core Q/K/V stage, and results in page-locked memory."""
import numpy as np
import pytest

from ullis_b200 import cuda, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,time,min_rows", [(1, 1, 4096), (3, 31, 4096), (2, 33, 4096), (5, 127, 256), (3, 250, 256)])
def test_bits_equal_the_exact_path_at_ragged_lengths(oracle, monkeypatch, batch, time, min_rows):
    monkeypatch.setenv("ULLIS_CUDA_WS2_MIN_ROWS", str(min_rows))        # both forms of the GEMM
    rt = cuda.CudaRuntime(0)
    try:
        d, rng = 256, np.random.default_rng(time)
        x = rng.standard_normal(batch * time * d).astype(np.float32)
        f16 = lambda a: np.asarray(a, np.float32).astype(np.float16).view(np.uint16)
        lin = lambda: {"bits": rng.integers(0, 1 << 32, d * d // 32, dtype=np.uint32), "scale": f16(rng.uniform(0.005, 0.02, d)),
                       "bias": f16(0.01 * rng.standard_normal(d))}
        p = {m: f16(rng.uniform(0, 1, d)) for m in ("x_q", "x_k", "x_v")} | {m: lin() for m in "qkvo"}
        p["e"] = f16(0.02 * rng.standard_normal(d))
        rt.kernel_timing(True)
        fast = rt.rosa_block_forward(x, p, batch, time, d)
        assert "gemm_qkv_signbits" in rt.kernel_times()
        rt.set_mode(cuda.MODE_EXACT)
        exact = rt.rosa_block_forward(x, p, batch, time, d)
        for name in ("q_plane", "k_plane", "v_plane", "idx"):
            assert np.array_equal(fast[name], exact[name]), name
        assert np.abs(fast["out"] - exact["out"]).max() <= 1e-2 * np.abs(exact["out"]).max()
    finally:
        rt.close()


def test_results_stay_apart_and_their_memory_comes_back(cuda_rt):
    x = np.arange(50_000, dtype=np.float32)
    first, second = cuda_rt.residual_add(x, x), cuda_rt.residual_add(x, -x)
    assert np.array_equal(first, 2 * x) and not second.any()            # two results alive at once
    held = cuda._RESULTS._held
    view = first[10:20].copy(), first[10:20]
    del first, second
    for _ in range(20):
        cuda_rt.residual_add(x, x)
    assert cuda._RESULTS._held <= held + 2 * cuda._RESULTS._block_size(x.nbytes)
    assert np.array_equal(view[0], view[1])                             # a view keeps its block
    small = cuda._ResultPool(limit=1 << 20)
    kept = [small.empty(cuda_rt, 100_000, np.float32) for _ in range(4)]   # beyond the limit: ordinary arrays
    assert small._held <= 1 << 20 and all(a.size == 100_000 for a in kept)
