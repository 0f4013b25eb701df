"""Every form of the one-kernel generation step (rows by warps of their own, wide CTAs, neither) with clusters that are not full, against
the step as separate kernels, bit for bit."""
import numpy as np
import pytest

from ullis_b200 import cuda, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,batches", [((512, 1, 512, 64, 2048), (10, 11, 19, 22, 27, 33, 39, 61, 127, 130)), ((256, 2, 300, 64, 512), (10, 23, 70)),
                                           ((1024, 1, 512, 64, 2048), (3, 9, 30)), ((128, 2, 300, 64, 256), (13, 75, 200))])
def test_forms_of_the_step(cuda_rt, monkeypatch, shape, batches):
    m = cuda.CudaHeron(cuda_rt, synth.heron_checkpoint(shape, batch_size=1, ln_gain_one=True))
    for batch in batches:
        tokens = synth.zipf_tokens(batch, 4 * batch, m.vocab_size).reshape(4, batch)
        one = m.generate_state(batch)
        monkeypatch.setenv("ULLIS_CUDA_GEN_UNFUSED", "1")
        plain = m.generate_state(batch)
        monkeypatch.delenv("ULLIS_CUDA_GEN_UNFUSED")
        for t in range(4):
            assert np.array_equal(one.step(tokens[t]), plain.step(tokens[t])), (batch, t)
        one.close()
        plain.close()
    m.close()
