"""GPU parity of the one-block digest's shortened first and last rounds: raw leaves on
both sides of 72 bytes and of the rate, aligned or not, hashed by a thread per leaf,
per pair of leaves and per four leaves, against the CPU oracle's roots."""
import pytest

import apple_b200 as azk
from tests import generators as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length,stride", [(0, 1), (1, 3), (63, 64), (64, 64), (64, 65), (71, 72), (71, 71), (72, 72), (79, 80), (128, 129), (135, 136), (136, 136), (136, 137)])
@pytest.mark.parametrize("treelet", [7, 8, 10])
def test_raw_leaves_by_threads(ctx, oracle, length, stride, treelet):
    n = 1 << 11
    leaves = G.make_leaves(n, stride, length, salt=length + treelet)
    plan = azk.SHA3RawLeavesMerkleCommitPlan(ctx, n, stride, length, treelet_log=treelet)
    assert plan.commit(leaves) == oracle.merkle_root(leaves, n, stride, length)


@pytest.mark.parametrize("log_count", [9, 10, 12, 13])
def test_prehashed_by_threads(ctx, oracle, log_count):
    d = G.make_leaves(1 << log_count, 32, 32, salt=log_count)
    assert azk.SHA3PrehashedLeavesMerkleCommitPlan(ctx, 1 << log_count).commit(d) == oracle.merkle_root_prehashed(d)
