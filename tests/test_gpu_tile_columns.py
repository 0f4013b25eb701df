"""Tiles of 32, 64 and 128 columns: broken last tiles of rows and columns against 64-bit sums, and rows that are alone in a call
against the same rows among enough others for wide tiles, bit for bit."""
import numpy as np
import pytest

from conftest import unpack_plane

pytestmark = pytest.mark.gpu


def f16(x):
    return np.asarray(x, np.float32).astype(np.float16).view(np.uint16)


# tiles of 128 columns: 1, 4 and 37 (32 columns), 38 and 74 (64 columns), 75 (128 columns)
@pytest.mark.parametrize("rows,K,N", [(1, 64, 8), (77, 128, 40), (128, 512, 512), (129, 576, 104), (4600, 64, 128), (4740, 64, 96), (4740, 128, 128), (9472, 64, 72),
                                      (9473, 64, 128)])
def test_linears_of_every_tile_width(cuda_rt, rows, K, N):
    rng = np.random.default_rng([rows, K, N])
    x = rng.standard_normal((rows, K), np.float32).astype(np.float16).astype(np.float32)
    bits = rng.integers(0, 2 ** 32, K * N // 32, dtype=np.uint32)
    scale, bias = f16(rng.uniform(0.005, 0.02, N)), f16(0.01 * rng.standard_normal(N))
    w = f16(rng.standard_normal(N * K) / np.sqrt(K))
    signs = 2.0 * unpack_plane(bits, N * K).reshape(N, K).astype(np.float64) - 1.0
    s, b = (a.view(np.float16).astype(np.float64) for a in (scale, bias))
    dense = w.view(np.float16).astype(np.float64).reshape(N, K)
    got = np.asarray(cuda_rt.binary_linear(x.ravel(), bits, scale, bias, rows, K, N)).reshape(rows, N)
    # exact products, K f32 additions and the two of scale and bias
    size = np.abs(x).astype(np.float64).sum(1)[:, None]
    assert (np.abs(got - (b + s * (x.astype(np.float64) @ signs.T))) <= (K + 2) * 2.0 ** -23 * (s * size + np.abs(b))).all()
    got16 = np.asarray(cuda_rt.fp16_linear(x.ravel(), w, rows, K, N)).reshape(rows, N)
    size16 = np.abs(x).astype(np.float64) @ np.abs(dense).T
    assert (np.abs(got16 - x.astype(np.float64) @ dense.T) <= (K + 2) * 2.0 ** -23 * size16).all()
    # among more rows
    more = np.concatenate([x, rng.standard_normal((128 * 160, K), np.float32).astype(np.float16).astype(np.float32)])
    assert np.array_equal(np.asarray(cuda_rt.binary_linear(more.ravel(), bits, scale, bias, len(more), K, N)).reshape(-1, N)[:rows], got)
    assert np.array_equal(np.asarray(cuda_rt.fp16_linear(more.ravel(), w, len(more), K, N)).reshape(-1, N)[:rows], got16)


@pytest.mark.parametrize("T", [31, 160, 500, 700, 1300])
def test_a_sequence_alone_and_among_others(cuda_rt, T):
    """The model's products: Q/K/V, O, key and value in tiles of other widths than in a batch, the same losses."""
    from ullis_b200 import cuda, synth
    m = cuda.CudaHeron(cuda_rt, synth.heron_checkpoint("small" if T <= 500 else "default", batch_size=24, ln_gain_one=True))
    tokens = np.random.default_rng(T).integers(0, m.vocab_size, 24 * T).astype(np.uint32)
    rows = m.forward_ce(tokens, tokens, cuda.CE_NO_IGNORE, 24, T, want_row_loss=True)[3]
    for b in (0, 23):
        one = tokens[b * T:(b + 1) * T]
        assert np.array_equal(m.forward_ce(one, one, cuda.CE_NO_IGNORE, 1, T, want_row_loss=True)[3], rows[b * T:(b + 1) * T])
    m.close()
