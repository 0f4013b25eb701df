"""The generation step as one cluster kernel against the step as separate kernels, bit for bit, at batch sizes that fill
clusters partly, need several sequences per cluster, fewer CTAs per cluster or several rounds."""
import numpy as np
import pytest

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
