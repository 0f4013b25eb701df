"""Calls whose streams are uneven or repeat themselves, so that the latest positions leave most of them to the contexts: a few or many
streams left, in one, two and four pieces, against the oracle's pushes."""
import numpy as np
import pytest

from conftest import pack_plane

pytestmark = pytest.mark.gpu


def bits(kind, T, n, rng):
    """[T, n] of q, k and v."""
    if kind == "biased":                                   # nine ones in ten
        return [(rng.random((T, n)) < 0.9).astype(np.uint8) for _ in range(3)]
    if kind == "slow":                                     # runs of about 20 steps
        return [(np.cumsum(rng.random((T, n)) < 0.05, axis=0) & 1).astype(np.uint8) for _ in range(3)]
    if kind == "periodic":
        phase = np.arange(T)[:, None] % rng.integers(16, 257, n)[None, :]
        base = rng.integers(0, 2, (2, 256, n), dtype=np.uint8)
        return [np.take_along_axis(base[i], phase, 0) for i in (0, 0, 1)]
    return [rng.integers(0, 2, (T, n), dtype=np.uint8) for _ in range(3)]


@pytest.mark.parametrize("T,B,C", [(40, 3, 256), (300, 3, 256), (700, 3, 512), (1023, 9, 512), (1100, 5, 512), (2048, 5, 512)])
@pytest.mark.parametrize("kind,share", [("biased", 1.0), ("slow", 1.0), ("periodic", 1.0), ("biased", 0.3), ("slow", 0.01)])
def test_streams_that_are_left(cuda_rt, oracle, T, B, C, kind, share):
    rng = np.random.default_rng([T, C, len(kind)])
    mine = rng.random(B * C) < share
    planes = []
    for x, even in zip(bits(kind, T, B * C, rng), bits("even", T, B * C, rng)):
        x = np.where(mine[None, :], x, even).astype(np.uint8)
        planes.append(pack_plane(x.reshape(T, B, C).transpose(1, 0, 2).reshape(B * T, C)))
    cuda_rt.kernel_timing(True)
    idx, _ = cuda_rt.rosa_qkv_1bit_fwd(*planes, np.zeros(C, np.uint16), B, T, C)
    ran = cuda_rt.kernel_times()
    cuda_rt.kernel_timing(False)
    assert 2 * cuda_rt.sam_counts()["automaton"] > B * C   # the listed streams: most, so the latest positions have run
    assert "rosa_context_left" in ran and ("rosa_context_left_many" in ran) == (T >= 700)
    assert np.array_equal(idx, oracle.rosa_qkv_batch_packed(*planes, B, T, C))


@pytest.mark.parametrize("T,B,C", [(127, 4, 512), (128, 2, 320), (300, 4, 512), (511, 8, 512)])
@pytest.mark.parametrize("kind,share", [("biased", 1.0), ("slow", 0.5), ("slow", 0.03)])
def test_few_short_streams_of_which_some_are_uneven(cuda_rt, oracle, T, B, C, kind, share):
    """More or fewer of them than the share from which on all streams go by contexts, and a length where they are not counted; two calls, since
    the count of one must not be the next one's."""
    test_streams_that_are_left(cuda_rt, oracle, T, B, C, kind, share)
    test_streams_that_are_left(cuda_rt, oracle, T, B, C, "even", 0.0)
