"""A wait of the generation step's kernel that runs out: the step fails with the timeout's status, every copy that is on its way
has landed, and the device goes on as before."""
import numpy as np
import pytest

from ullis_b200 import cuda, synth

pytestmark = pytest.mark.gpu

DEFAULT, ODD = (512, 2, 8192, 64, 2048), (64, 2, 300, 80, 256)


# One sequence per cluster of 16 (one sum per lane), several sequences and the ring, several rounds of clusters; no poll at all,
# and few of them: whether and where a wait runs out is then a matter of time.
@pytest.mark.parametrize("shape,batch", [(DEFAULT, 1), (DEFAULT, 8), (DEFAULT, 64), (ODD, 5), (ODD, 150)])
@pytest.mark.parametrize("polls", [0, 1, 3, 20])
def test_a_wait_that_runs_out(cuda_rt, monkeypatch, shape, batch, polls):
    m = cuda.CudaHeron(cuda_rt, synth.heron_checkpoint(shape, batch_size=1, ln_gain_one=True))
    tokens = synth.zipf_tokens(batch, 3 * batch, m.vocab_size).reshape(3, batch)
    good = m.generate_state(batch)
    expected = [good.step(t).copy() for t in tokens]
    monkeypatch.setenv("ULLIS_CUDA_GEN_WAIT_POLLS", str(polls))
    short = m.generate_state(batch)
    monkeypatch.delenv("ULLIS_CUDA_GEN_WAIT_POLLS")
    for _ in range(3):
        short.reset()
        try:
            for t, logits in zip(tokens, expected):
                assert np.array_equal(short.step(t), logits)
            assert polls > 0
        except cuda.UllisCudaError as e:
            assert e.code == cuda.ERR_TIMEOUT
            with pytest.raises(cuda.UllisCudaError, match="unusable after a failed step"):
                short.step(tokens[0])
            x = np.arange(8, dtype=np.float32)
            assert np.array_equal(cuda_rt.residual_add(x, x), 2 * x)
        good.reset()
        for t, logits in zip(tokens, expected):
            assert np.array_equal(good.step(t), logits)
    good.close()
    short.close()
    m.close()
