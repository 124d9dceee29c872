"""GPU parity of the several-rounds-a-launch folds with the CPU oracle: tiles that end
inside the input, chains of one, eleven, twelve and more rounds, counts that are not
powers of two, M31 (canonical domain) and QM31 inverse layers."""
import numpy as np
import pytest

import apple_b200 as azk
from tests import generators as G

pytestmark = pytest.mark.gpu


def _values(rng, n):
    return rng.integers(0, G.P, size=(n, 4), dtype=np.uint32)


@pytest.mark.parametrize("log_size,rounds", [(1, 1), (10, 10), (11, 1), (11, 11), (12, 11), (12, 12), (14, 5), (15, 13), (17, 17)])
def test_circle_chain(ctx, oracle, log_size, rounds):
    rng = np.random.default_rng(100 * log_size + rounds)
    ev, ch = _values(rng, 1 << log_size), _values(rng, rounds)
    ev[:2] = G.P - 1  # largest canonical limbs
    ch[0] = G.P - 1
    plan = azk.CircleFRIFoldChainPlan(ctx, log_size, rounds)
    assert np.array_equal(plan.execute(ev, ch), oracle.circle_fold_chain(log_size, ev, ch))


@pytest.mark.parametrize("count,rounds", [(2, 1), (6, 1), (3 * 2048, 11), (5 * 4096, 12), (1000, 3), (2050, 1), (2048 + 64, 6), (1 << 13, 13)])
def test_qm31_chain_of_any_even_count(ctx, oracle, count, rounds):
    rng = np.random.default_rng(count + rounds)
    ev, ch = _values(rng, count), _values(rng, rounds)
    layers = [_values(rng, count >> (r + 1)) | 1 for r in range(rounds)]
    for l in layers:
        l[l >= G.P] = 1
    want = ev
    for inv, c in zip(layers, ch):
        want = oracle.fold(want, inv, c)
    assert np.array_equal(azk.QM31FRIFoldChainPlan(ctx, count, rounds).execute(ev, layers, ch), want)
