"""The generation step as one cluster kernel against the step as separate kernels, bit for bit, at batch sizes that fill
clusters partly, need several sequences per cluster, fewer CTAs per cluster or several rounds."""
import numpy as np
import pytest

from conftest import pack_streams
from ullis_b200 import cuda, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,batches,steps", [("small", (1, 3, 9, 31, 77), 70), ((64, 2, 300, 80, 256), (1, 5, 150), 70),
                                                 ((512, 1, 8192, 64, 2048), (2, 8, 17, 64), 6)])
def test_one_kernel_equals_separate_kernels(cuda_rt, monkeypatch, shape, batches, steps):
    m = cuda.CudaHeron(cuda_rt, synth.heron_checkpoint(shape, batch_size=1, ln_gain_one=True))
    for batch in batches:
        tokens = synth.zipf_tokens(batch, steps * batch, m.vocab_size).reshape(steps, batch)
        one = m.generate_state(batch)
        monkeypatch.setenv("ULLIS_CUDA_GEN_UNFUSED", "1")
        plain = m.generate_state(batch)
        monkeypatch.delenv("ULLIS_CUDA_GEN_UNFUSED")
        cuda_rt.kernel_timing(True)
        one.step(tokens[0])
        assert list(cuda_rt.kernel_times())[-1] == "gen_step"
        cuda_rt.kernel_timing(False)
        one.reset()
        for t in range(steps):
            assert np.array_equal(one.step(tokens[t]), plain.step(tokens[t])), (batch, t)
        one.close()
        plain.close()
    m.close()


@pytest.mark.parametrize("T,n,run", [(1100, 70, 40), (2300, 64, 150), (4500, 12, 1500)])
def test_pushes_of_streams_that_hardly_ever_change(cuda_rt, oracle, T, n, run):
    """Runs of equal bits longer than 32 steps, many of the same length: the search by runs, at word and chunk borders."""
    rng = np.random.default_rng(T)
    lengths = rng.choice([run // 3, run, run, 32 * (run // 32 + 1)], (3, n, 1 + T // max(run // 3, 1)))
    bits = np.zeros((3, n, T), np.uint8)
    for a in range(3):
        for s in range(n):
            level = rng.random(lengths.shape[2]) < 0.8
            # a short interruption between the runs, so that runs of one bit follow on each other
            row = np.concatenate([np.r_[np.full(m, b), np.full(rng.integers(1, 3), not b)] for m, b in zip(lengths[a, s], level)])
            bits[a, s] = row[:T]
    bits[0, ::5] = bits[0, ::5, :1]                      # a constant query
    bits[1, 3::7] = bits[0, 3::7]                        # keys like the queries
    words = oracle.rosa_qkv_streams(*(pack_streams(b) for b in bits), n, T)
    ref = np.unpackbits(words.view(np.uint8).reshape(n, -1), axis=1, bitorder="little")[:, :T].T
    p = cuda.CudaRosaPushers(cuda_rt, n, T)
    assert np.array_equal(p.push(*(b.T for b in bits)), ref)
    p.close()
