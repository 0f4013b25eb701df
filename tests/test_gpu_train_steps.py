"""Optimiser kernels of a training step at the edges of their shares: rows of a packed matrix in more than one round or fewer
words than a warp takes, gradient products in shares, tokens with whole batches of occurrences and without."""
import pytest

import test_gpu_train as base

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
