"""Kernels of a training step at the edges of their shares: rows of a packed matrix in more than one round or fewer words than
a warp takes, gradient products in shares, tokens with whole batches of occurrences and without; the CMix gradient and its
operands in one kernel."""
import numpy as np
import pytest

import test_gpu_train as base
from ullis_b200 import checkpoint as ckpt
from ullis_b200 import cuda, synth

pytestmark = pytest.mark.gpu

CASES = {
    "rows-of-640": ((640, 1, 260, 70, 640), 1, 70, 0.05, 2),
    "rows-of-96": ((96, 1, 260, 33, 96), 2, 33, 0.05, 2),
    "product-in-shares": ((256, 1, 260, 1024, 256), 2, 1024, 0.005, 1),
}


@pytest.mark.parametrize("case", CASES)
def test_steps_match_the_cpu_restatement_at_the_edges(cuda_rt, oracle, case, monkeypatch):
    monkeypatch.setitem(base.CASES, case, CASES[case])
    base.test_steps_match_the_cpu_restatement(cuda_rt, oracle, case, "fast")


def _one_step(checkpoint, batch, time, min_rows, monkeypatch):
    """Loss and stepped tensors, or the error, with the pair form of the matrix products from `min_rows` rows on."""
    monkeypatch.setenv("ULLIS_CUDA_WS2_MIN_ROWS", str(min_rows))
    rt = cuda.CudaRuntime(0)
    try:
        model = cuda.CudaHeron(rt, checkpoint)
        train = model.train_state()
        tokens = synth.zipf_tokens(9, batch * time, 260)
        rt.kernel_timing(True)
        loss = train.train_step(tokens, tokens, cuda.CE_NO_IGNORE, batch, time, 0.005)["loss"]
        fused = "gemm_cmix_grad" in rt.kernel_times()
        rt.kernel_timing(False)
        values = {name: base_value(train, name, n) for name, n in
                  (("blocks.0.ffn.key.latent", 64 * 2048), ("blocks.0.ffn.value", 64 * 2048), ("blocks.0.ffn.x_k", 64))}
        return fused, loss, values
    except cuda.UllisCudaError as e:
        return None, e.code, "FP16 range" in str(e)


def base_value(train, name, n):
    return train.read(name, np.uint16, n).view(np.float16).astype(np.float32) + train.read(name + ".residual", np.float32, n)


@pytest.mark.parametrize("batch,time,head_scale", [(3, 700, None), (3, 683, None), (3, 700, 4000.0), (3, 700, 8000.0), (3, 700, 16000.0)])
def test_cmix_gradient_and_its_operands_in_one_kernel(batch, time, head_scale, monkeypatch):
    """Rows that end inside a tile and inside the padding of the transposes; gradients that leave the range of FP16 are reported.
    The two routes form the same FP16 operands from the same f32 product: the stepped tensors agree within the tolerance of a
    gradient (GRAD_TOL x learning rate), the loss to rounding."""
    cfg = synth.train_config(64, 1, 260, 700, 3, 2048)
    tensors = synth.heron_tensors(cfg, seed=4, ln_gain_one=True)
    if head_scale:
        tensors["head.scale"] = synth.f16_bits(np.full(260, head_scale))
        for name, factor in (("blocks.0.ffn.value", 25.0),):
            tensors[name] = synth.f16_bits(tensors[name].view(np.float16).astype(np.float64) * factor)
    checkpoint = ckpt.to_safetensors_bytes(tensors, cfg, step=0)
    fused, loss, values = _one_step(checkpoint, batch, time, 1, monkeypatch)
    apart, loss_apart, values_apart = _one_step(checkpoint, batch, time, 1 << 30, monkeypatch)
    if fused is None or apart is None:
        assert (fused, loss, values) == (apart, loss_apart, values_apart) and values
        return
    assert fused and not apart
    assert abs(loss - loss_apart) <= 1e-5 * abs(loss)
    for name in values:
        assert np.abs(values[name] - values_apart[name]).max() <= 0.005 * base.GRAD_TOL, name
