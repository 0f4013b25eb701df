"""The shapes on which the forms of the one-kernel generation step are compared with the separate kernels do run as one kernel: otherwise
that comparison is of the separate kernels with themselves."""
import pytest

from test_gpu_generate_shapes import test_forms_of_the_step as forms
from ullis_b200 import cuda, synth

pytestmark = pytest.mark.gpu

SHAPES = next(mark for mark in forms.pytestmark if mark.name == "parametrize").args[1]


@pytest.mark.parametrize("shape,batches", SHAPES)
def test_the_step_is_one_kernel(cuda_rt, shape, batches):
    m = cuda.CudaHeron(cuda_rt, synth.heron_checkpoint(shape, batch_size=1, ln_gain_one=True))
    for batch in batches:
        state = m.generate_state(batch)
        cuda_rt.kernel_timing(True)
        state.step(synth.zipf_tokens(batch, batch, m.vocab_size))
        ran = list(cuda_rt.kernel_times())
        cuda_rt.kernel_timing(False)
        assert [name for name in ran if "_" in name] == ["gen_step"], (batch, ran)
        state.close()
    m.close()
