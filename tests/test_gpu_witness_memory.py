"""A witness plan takes its device memory when it is made: no call of any length or
form allocates more, so none can fail for memory that its creation did not fail for."""
import numpy as np
import pytest
import torch

import apple_b200 as azk
from tests import generators as G

pytestmark = pytest.mark.gpu


def _calls(plan, log_size):
    rng = np.random.default_rng(log_size)
    n = 1 << (log_size - 1)
    for count in (n, 3, min(n, 5000), n // 2 + 1, n):
        for lifted in (False, True):
            x, y = (rng.integers(0, G.P, size=(count, 4), dtype=np.uint32) for _ in range(2))
            if lifted:
                x[:, 1:] = 0
                y[:, 1:] = 0
            plan.execute(x, y)
            yield torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("log_size,most", [(13, 16 << 20), (18, 64 << 20), (20, 192 << 20), (22, 640 << 20)])
def test_calls_allocate_nothing(ctx, log_size, most):
    list(_calls(azk.CircleWitnessToFFTBasisPlan(ctx, log_size), log_size))  # the kernels' own memory
    before = torch.cuda.mem_get_info()[0]
    plan = azk.CircleWitnessToFFTBasisPlan(ctx, log_size)
    made = torch.cuda.mem_get_info()[0]
    assert 0 < before - made <= most
    assert all(free == made for free in _calls(plan, log_size))
