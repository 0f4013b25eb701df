"""Few listed streams among constant ones: two or more CTAs take the steps of a stream in parts (two, three and four of them), streams
that go by bits, by runs, and to the sets of lags, in calls that the latest positions could take too."""
import numpy as np
import pytest

from conftest import pack_plane
from test_gpu_rosa_match import planes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["even", "biased", "repeating"])
@pytest.mark.parametrize("T,B,C,listed", [(33, 1, 256, 5), (64, 1, 256, 70), (300, 2, 256, 60), (512, 1, 128, 40), (513, 1, 256, 130), (1023, 3, 256, 90),
                                          (2048, 1, 512, 73), (2047, 2, 512, 49), (2048, 1, 64, 1), (4100, 1, 128, 30), (8192, 1, 64, 12)])
def test_parts_of_streams(cuda_rt, oracle, kind, T, B, C, listed):
    rng = np.random.default_rng([T, B * C, listed])
    q, k, v = (np.asarray(x, np.uint8).copy() for x in planes(kind, T, B * C, rng))
    constant = np.ones(B * C, bool)
    constant[rng.choice(B * C, listed, replace=False)] = False
    k[:, constant] = rng.integers(0, 2, constant.sum())
    q, k, v = (pack_plane(x.reshape(T, B, C).transpose(1, 0, 2).reshape(B * T, C)) for x in (q, k, v))
    want = oracle.rosa_qkv_batch_packed(q, k, v, B, T, C)
    for _ in range(2):
        idx, _ = cuda_rt.rosa_qkv_1bit_fwd(q, k, v, np.zeros(C, np.uint16), B, T, C)
        assert np.array_equal(idx, want)
