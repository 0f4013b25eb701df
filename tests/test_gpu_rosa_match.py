"""The automaton-free ROSA match (lookup by contexts and by run lengths, sets of lags, constant q) against the oracle's
pushes: lengths around its word, piece and set-width limits, and streams that each of its ways has to take."""
import numpy as np
import pytest

from conftest import pack_plane
from ullis_b200 import cuda

pytestmark = pytest.mark.gpu


def planes(kind, T, C, rng):
    if kind == "even":
        return [rng.integers(0, 2, (T, C), dtype=np.uint8) for _ in range(3)]
    if kind == "biased":        # q and k biased independently: by bits, by runs, or neither
        p = rng.choice([0.002, 0.03, 0.1, 0.2, 0.5, 0.8, 0.93, 0.99], (3, 1, C))
        return [(rng.random((T, C)) < p[i]).astype(np.uint8) for i in range(3)]
    if kind == "repeating":     # long agreements: sets of lags, windows longer than the ring
        period = rng.integers(2, 100, C)
        base = rng.integers(0, 2, (2, 100, C), dtype=np.uint8)
        phase = np.arange(T)[:, None] % period[None, :]
        q, v = (np.take_along_axis(base[i], phase, 0) for i in range(2))
        return [q ^ (rng.random((T, C)) < 0.002), q ^ (rng.random((T, C)) < 0.001), v ^ (rng.random((T, C)) < 0.3)]
    q, k, v = (rng.integers(0, 2, (T, C), dtype=np.uint8) for _ in range(3))
    q[:] = rng.integers(0, 2, (1, C))                                   # constant q, keys of several densities
    return [q, (rng.random((T, C)) < rng.choice([0.01, 0.5, 0.99], (1, C))).astype(np.uint8), v]


@pytest.mark.parametrize("kind", ["even", "biased", "repeating", "constant_q"])
@pytest.mark.parametrize("T", [2, 32, 63, 64, 65, 127, 513, 1023, 1025, 2048, 2049, 4097, 8191, 8192])
def test_match_equals_the_pushes(cuda_rt, oracle, kind, T):
    C = 96 if T <= 2049 else 32
    rng = np.random.default_rng([T, len(kind)])
    q, k, v = (pack_plane(np.asarray(x, np.uint8)) for x in planes(kind, T, C, rng))
    cuda_rt.kernel_timing(True)
    idx, _ = cuda_rt.rosa_qkv_1bit_fwd(q, k, v, np.zeros(C, np.uint16), 1, T, C)
    ran = cuda_rt.kernel_times()
    cuda_rt.kernel_timing(False)
    assert "rosa_context" in ran and "rosa_match" in ran
    assert np.array_equal(idx, oracle.rosa_qkv_batch_packed(q, k, v, 1, T, C))


@pytest.mark.parametrize("T,B,C,left", [(1024, 1, 96, 0.3), (8192, 1, 32, 0.4), (300, 9, 128, 0.2), (700, 9, 128, 0.3), (700, 9, 128, 0.9),
                                        (1100, 5, 256, 0.2), (1100, 5, 256, 0.8), (1030, 9, 256, 0.3)])
def test_each_split_of_the_contexts(cuda_rt, oracle, T, B, C, left):
    """Few or most streams without a closed form, in few and in many streams: every shape of the context kernel."""
    rng = np.random.default_rng([T, B])
    q, k, v = planes("biased", T, B * C, rng)
    q, k, v = (x.reshape(T, B, C).transpose(1, 0, 2).copy() for x in (q, k, v))
    k[:, :, rng.random(C) >= left] = 1          # the others: constant keys
    q, k, v = (pack_plane(x.reshape(B * T, C)) for x in (q, k, v))
    idx, _ = cuda_rt.rosa_qkv_1bit_fwd(q, k, v, np.zeros(C, np.uint16), B, T, C)
    assert np.array_equal(idx, oracle.rosa_qkv_batch_packed(q, k, v, B, T, C))


# Beside those: fewer streams than SMs, the steps and streams where a shape changes, and lengths that leave an SM two or
# one block of 256 threads (512 or 1024 threads take every stream there).
@pytest.mark.parametrize("T,B,C,left", [(511, 2, 64, 0.9), (512, 2, 64, 0.9), (513, 1, 148, 0.9), (513, 1, 149, 0.9), (511, 3, 256, 0.9), (1023, 3, 256, 0.3),
                                        (1023, 3, 256, 0.9), (2048, 1, 148, 0.2), (2048, 9, 256, 0.2), (2048, 9, 256, 0.9), (6000, 5, 64, 0.2), (6000, 5, 64, 0.9),
                                        (7000, 5, 256, 0.9), (7000, 9, 256, 0.04), (8192, 3, 64, 0.9), (8192, 9, 256, 0.04)])
def test_each_choice_of_shape(cuda_rt, oracle, T, B, C, left):
    test_each_split_of_the_contexts(cuda_rt, oracle, T, B, C, left)


def test_two_runtimes_of_one_device_at_lengths_of_their_own(oracle):
    """Shared memory of the context kernel grows with the length, its limit belongs to the function: a runtime at a short
    length takes nothing away from one at a long length."""
    runtimes = [cuda.CudaRuntime(0) for _ in range(2)]
    try:
        for which, T, C in ((0, 8192, 32), (1, 64, 32), (0, 8192, 32), (1, 512, 64), (1, 8192, 32), (0, 4096, 32), (1, 8192, 32)):
            q, k, v = (pack_plane(x) for x in planes("even", T, C, np.random.default_rng([T, which])))
            idx, _ = runtimes[which].rosa_qkv_1bit_fwd(q, k, v, np.zeros(C, np.uint16), 1, T, C)
            assert np.array_equal(idx, oracle.rosa_qkv_batch_packed(q, k, v, 1, T, C)), (which, T)
    finally:
        for rt in runtimes:
            rt.close()
