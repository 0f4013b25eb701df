"""Op-level calls with large results run in shares, with the copies beside the kernels: the same results as the shares by
themselves, at sizes that cut unevenly, with results in page-locked and in ordinary memory."""
import numpy as np
import pytest

from ullis_b200 import cuda, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 255, 513, 1100])
def test_packed_linear_in_shares(cuda_rt, rows):
    K, N = 128, 4096                                  # 513 rows: two shares, 1100: four
    rng = np.random.default_rng(rows)
    x = rng.standard_normal((rows, K), np.float32)
    bits = rng.integers(0, 1 << 32, K * N // 32, dtype=np.uint32)
    scale, bias = (synth.f16_bits(rng.uniform(0.01, 0.02, N)) for _ in range(2))
    whole = cuda_rt.binary_linear(x.ravel(), bits, scale, bias, rows, K, N).reshape(rows, N)
    for r in range(0, rows, 200):
        part = x[r:r + 200]
        assert np.array_equal(whole[r:r + 200].ravel(), cuda_rt.binary_linear(part.ravel(), bits, scale, bias, len(part), K, N))


@pytest.mark.parametrize("B,T,C", [(5, 1000, 512), (9, 513, 1024), (3, 8192, 1024), (7, 333, 1000)])
def test_rosa_in_shares(cuda_rt, B, T, C):
    rng = np.random.default_rng([B, T])
    words = (B * T * C + 31) // 32
    planes = [rng.integers(0, 1 << 32, words, dtype=np.uint32) for _ in range(3)]
    if T == 513:
        planes[1][: words // 2] = 0                   # half of the streams have constant keys
    e = synth.f16_bits(rng.standard_normal(C))
    idx, out = cuda_rt.rosa_qkv_1bit_fwd(*planes, e, B, T, C)
    counts = cuda_rt.sam_counts()
    listed = 0
    if T * C % 32 == 0:
        per = T * C // 32
        for b in range(B):
            one, o = cuda_rt.rosa_qkv_1bit_fwd(*(p[b * per:(b + 1) * per] for p in planes), e, 1, T, C)
            assert np.array_equal(one, idx[b * T * C:(b + 1) * T * C]) and np.array_equal(o, out[b * T * C:(b + 1) * T * C]), b
            listed += cuda_rt.sam_counts()["automaton"]
        assert counts["total"] == B * C and counts["automaton"] == listed
    kept, _ = cuda_rt.rosa_qkv_1bit_fwd(*planes, e, B, T, C, want_out=False)
    assert np.array_equal(kept, idx)


def test_a_call_whose_kernels_are_timed_goes_in_one_piece(cuda_rt):
    """The times are then those of the kernels, not of waits for a share's copies."""
    rows, K, N = 2048, 512, 2048
    rng = np.random.default_rng(5)
    x = rng.standard_normal(rows * K, np.float32)
    bits = rng.integers(0, 1 << 32, K * N // 32, dtype=np.uint32)
    scale = synth.f16_bits(rng.uniform(0.01, 0.02, N))
    shared = cuda_rt.binary_linear(x, bits, scale, scale, rows, K, N)
    cuda_rt.kernel_timing(True)
    whole = cuda_rt.binary_linear(x, bits, scale, scale, rows, K, N)
    times = cuda_rt.kernel_times()
    cuda_rt.kernel_timing(False)
    assert [n for name, (_, n) in times.items() if name.startswith("gemm_")] == [1]
    assert np.array_equal(whole, shared)
