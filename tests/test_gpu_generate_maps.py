"""Generation states made and closed in turn: the tensor maps of a state's value weights lie in device memory that the state
before it gave back, with boxes and weights of its own."""
import numpy as np
import pytest

from ullis_b200 import cuda, synth

pytestmark = pytest.mark.gpu


def test_states_of_two_models_in_turn(cuda_rt, monkeypatch):
    steps, batches = 4, (1, 64, 8)
    models = [cuda.CudaHeron(cuda_rt, synth.heron_checkpoint(shape, batch_size=1, ln_gain_one=True))
              for shape in ((512, 2, 300, 64, 2048), (256, 3, 520, 64, 1024))]
    inputs, expected = {}, {}
    monkeypatch.setenv("ULLIS_CUDA_GEN_UNFUSED", "1")
    for i, m in enumerate(models):
        for batch in batches:
            inputs[i, batch] = synth.zipf_tokens(batch, steps * batch, m.vocab_size).reshape(steps, batch)
            plain = m.generate_state(batch)
            expected[i, batch] = [plain.step(t).copy() for t in inputs[i, batch]]
            plain.close()
    monkeypatch.delenv("ULLIS_CUDA_GEN_UNFUSED")
    for _ in range(3):
        for batch in batches:
            for i, m in enumerate(models):
                state = m.generate_state(batch)
                for t, tokens in enumerate(inputs[i, batch]):
                    assert np.array_equal(state.step(tokens), expected[i, batch][t]), (i, batch, t)
                state.close()
    for m in models:
        m.close()
