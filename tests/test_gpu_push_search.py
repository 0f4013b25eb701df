"""The search of a push by bit masks (rosa push kernels of the generation step) at the borders of words and of the 32 words of a warp:
positions of the first word with short histories, agreements of exactly 8, 9, 31 and 32 steps, the latest of equals."""
import numpy as np
import pytest

from conftest import pack_streams
from ullis_b200 import cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 40])      # few open streams: by the whole warp, many: a lane each
@pytest.mark.parametrize("T", [31, 33, 64, 70, 1023, 1025, 1090])
def test_agreements_at_borders(cuda_rt, oracle, T, n):
    rng = np.random.default_rng([T, n])
    q, k, v = (rng.integers(0, 2, (n, T), dtype=np.uint8) for _ in range(3))
    if T >= 64:
        for s in range(n):      # histories that agree over a chosen number of steps before a difference
            for _ in range(6):
                m, end = int(rng.choice([7, 8, 9, 31, 32, 33])), int(rng.integers(34, T))
                at = int(rng.choice([31, 32, 33, 62, 63, max(end - 2, 1)]))
                if at + 1 > m and at < end and end >= m:
                    q[s, end - m + 1:end + 1] = k[s, at - m + 1:at + 1]
                    q[s, end - m] = 1 - k[s, at - m]
    words = oracle.rosa_qkv_streams(pack_streams(q), pack_streams(k), pack_streams(v), n, T)
    ref = np.unpackbits(words.view(np.uint8).reshape(n, -1), axis=1, bitorder="little")[:, :T].T
    p = cuda.CudaRosaPushers(cuda_rt, n, T)
    assert np.array_equal(p.push(q.T, k.T, v.T), ref)
    p.close()
