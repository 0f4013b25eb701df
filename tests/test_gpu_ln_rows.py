"""LayerNorm + mix + 16-bit operands: every number of rows per warp gives the same losses, bit for bit."""
import numpy as np
import pytest

from ullis_b200 import cuda, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,batch,time", [(128, 7, 37), (512, 5, 33), (640, 3, 70), (1024, 2, 41)])
def test_rows_per_warp_give_the_same_losses(d, batch, time, monkeypatch):
    """Rows that end inside a warp's share, sequences that begin inside one, widths with and without loads ahead."""
    checkpoint = synth.heron_checkpoint((d, 2, 300, 128, 2 * d), batch_size=8, ln_gain_one=True)
    tokens = synth.uniform_tokens(d, batch * time, 300)
    losses = {}
    for per_warp in (1, 2, 3, 4, 8):
        monkeypatch.setenv("ULLIS_CUDA_LN_ROWS", str(per_warp))
        rt = cuda.CudaRuntime(0)
        model = cuda.CudaHeron(rt, checkpoint)
        losses[per_warp] = model.forward_ce(tokens, tokens, cuda.CE_NO_IGNORE, batch, time, want_row_loss=True)[3]
        model.close()
        rt.close()
    for per_warp in losses:
        np.testing.assert_array_equal(losses[per_warp], losses[1])
