"""The latest positions of contexts (rosa_heads.cuh), compiled for the host, against the oracle's pushes."""
import numpy as np
import pytest

from conftest import pack_streams
from test_rosa_match_host import rosa_host  # noqa: F401
from test_sam_core_host import _streams

HEADS = 5


@pytest.mark.parametrize("T", [1, 2, 3, 4, 5])
def test_every_input_of_a_few_steps(oracle, rosa_host, T):  # noqa: F811
    n = 1 << (3 * T)
    a = np.arange(n, dtype=np.uint32)
    m = (1 << T) - 1
    q, k, v = a & m, (a >> T) & m, (a >> (2 * T)) & m
    assert np.array_equal(rosa_host(HEADS, q, k, v, n, T), oracle.rosa_qkv_streams(q, k, v, n, T))


@pytest.mark.parametrize("kind", ["iid", "qk_same", "biased", "periodic", "periodic_clean", "q_const", "k_const"])
@pytest.mark.parametrize("T", [12, 31, 32, 33, 43, 65, 777, 2048, 2081, 4097, 8192])
def test_streams(oracle, rosa_host, kind, T):  # noqa: F811
    """Histories shorter than a context, rows that are not whole, contexts met in the row and before it, chains."""
    n = 400 if T <= 65 else 24 if T <= 2081 else 4
    rng = np.random.default_rng([T, n, 5])
    q, k, v = (pack_streams(np.asarray(b, np.uint8)) for b in _streams(kind, n, T, rng))
    assert np.array_equal(rosa_host(HEADS, q, k, v, n, T), oracle.rosa_qkv_streams(q, k, v, n, T))
