"""The latest positions of contexts (the first launch of the contexts) against the oracle's pushes: rows that are not whole, streams in one, two and
four pieces, pieces that end past the last row, and streams that have to be given up beside even ones."""
import numpy as np
import pytest

from conftest import pack_plane
from test_gpu_rosa_match import planes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B,C,odd", [(1, 9, 256, 0.0), (12, 9, 256, 0.2), (33, 3, 256, 0.2), (64, 40, 512, 0.1), (127, 3, 256, 0.3), (511, 3, 256, 0.3),
                                       (513, 3, 256, 0.3), (700, 16, 512, 0.1), (1023, 3, 256, 0.3), (1024, 5, 512, 0.2), (1025, 15, 512, 0.02),
                                       (1100, 5, 512, 0.4), (1531, 9, 256, 0.2), (2047, 5, 512, 0.2), (2048, 9, 256, 0.3), (1024, 72, 512, 0.0)])
def test_even_streams_beside_others(cuda_rt, oracle, T, B, C, odd):
    rng = np.random.default_rng([T, B, C])
    kinds = ["even", "biased", "repeating", "constant_q"]
    kind = rng.choice(4, B * C, p=[1 - odd, odd * 0.5, odd * 0.3, odd * 0.2])
    q, k, v = (x.astype(np.uint8) for x in planes("even", T, B * C, rng))
    for i in range(1, 4):
        mine = np.flatnonzero(kind == i)
        if len(mine):
            for x, y in zip((q, k, v), planes(kinds[i], T, len(mine), rng)):
                x[:, mine] = y
    q, k, v = (pack_plane(x.reshape(T, B, C).transpose(1, 0, 2).reshape(B * T, C)) for x in (q, k, v))
    cuda_rt.kernel_timing(True)
    idx, _ = cuda_rt.rosa_qkv_1bit_fwd(q, k, v, np.zeros(C, np.uint16), B, T, C)
    ran = cuda_rt.kernel_times()
    cuda_rt.kernel_timing(False)
    assert "rosa_context_left" in ran
    assert np.array_equal(idx, oracle.rosa_qkv_batch_packed(q, k, v, B, T, C))
