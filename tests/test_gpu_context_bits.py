"""Streams with evenly spread keys beside uneven ones in one launch: a CTA changes the number of context bits from stream to
stream (up to 4096 steps), in both shapes that do so."""
import numpy as np
import pytest

from conftest import pack_plane
from test_gpu_rosa_match import planes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B,C,left", [(300, 1, 290, 1.0), (700, 4, 256, 1.0), (1030, 8, 256, 0.4), (2047, 4, 512, 0.4), (2048, 3, 256, 1.0),
                                        (4096, 4, 256, 0.4), (4096, 1, 148, 1.0), (4097, 4, 256, 0.4)])
def test_even_and_uneven_streams_in_turn(cuda_rt, oracle, T, B, C, left):
    rng = np.random.default_rng([T, B, C])
    even, biased = planes("even", T, B * C, rng), planes("biased", T, B * C, rng)
    pick = np.arange(B * C) % 2 == 0
    q, k, v = (np.where(pick, e, b).astype(np.uint8) for e, b in zip(even, biased))
    k[:, rng.random(B * C) >= left] = 1          # constant keys: not listed
    q, k, v = (pack_plane(x.reshape(T, B, C).transpose(1, 0, 2).reshape(B * T, C)) for x in (q, k, v))
    idx, _ = cuda_rt.rosa_qkv_1bit_fwd(q, k, v, np.zeros(C, np.uint16), B, T, C)
    assert np.array_equal(idx, oracle.rosa_qkv_batch_packed(q, k, v, B, T, C))
