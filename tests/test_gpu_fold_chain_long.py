"""GPU parity of long fold chains with the CPU oracle: from 2^19 values on a launch
stops after five rounds, from 2^24 on twice, so inverse layers and the values between
launches start where the launch before ended.  M31 (canonical domain) and QM31 inverse
layers, resident and host forms, a count that is not a power of two."""
import numpy as np
import pytest

import apple_b200 as azk
from tests import generators as G

pytestmark = pytest.mark.gpu


def _values(rng, n):
    return rng.integers(0, G.P, size=(n, 4), dtype=np.uint32)


@pytest.mark.parametrize("log_size,rounds", [(19, 1), (19, 5), (19, 6), (20, 16), (20, 20), (24, 10), (24, 11), (24, 22)])
def test_circle_chain(ctx, oracle, log_size, rounds):
    rng = np.random.default_rng(100 * log_size + rounds)
    ev, ch = _values(rng, 1 << log_size), _values(rng, rounds)
    ev[-2:] = G.P - 1  # largest canonical limbs
    want = oracle.circle_fold_chain(log_size, ev, ch)
    plan = azk.CircleFRIFoldChainPlan(ctx, log_size, rounds)
    assert np.array_equal(plan.execute(ev, ch), want)
    if log_size < 24:
        src, dst = ctx.alloc(ev.nbytes), ctx.alloc(want.nbytes)
        src.upload(ev)
        plan.execute_resident(src.ptr, dst.ptr, ch)
        assert dst.download(want.nbytes) == want.tobytes()


@pytest.mark.parametrize("count,rounds", [(1 << 19, 6), (3 << 18, 1), (3 << 18, 5), (3 << 18, 18), ((1 << 19) + (1 << 12), 12), (1 << 20, 17), (5 << 22, 12)])
def test_qm31_chain(ctx, oracle, count, rounds):
    rng = np.random.default_rng(count + rounds)
    ev, ch = _values(rng, count), _values(rng, rounds)
    layers = [np.maximum(_values(rng, count >> (r + 1)), 1) for r in range(rounds)]
    want = ev
    for inv, c in zip(layers, ch):
        want = oracle.fold(want, inv, c)
    assert np.array_equal(azk.QM31FRIFoldChainPlan(ctx, count, rounds).execute(ev, layers, ch), want)
