"""GPU parity of the commit kernel's three hashing forms (a pair of lanes, one
thread, a warp per permutation) where they meet: treelets of half, one, two and
four times the CTA's threads, groups on both sides of eight nodes, and trees down to
a single leaf, against the CPU oracle's proof bytes and chains."""
import numpy as np
import pytest

import apple_b200 as azk
from tests import generators as G

pytestmark = pytest.mark.gpu
PUB = bytes(range(32))


def _evaluations(n, seed):
    return np.random.default_rng(seed).integers(0, (1 << 31) - 1, (n, 4), dtype=np.uint32)


@pytest.mark.parametrize("threads", [128, 256, 512])
@pytest.mark.parametrize("ratio_log,group_log", [(-1, 1), (-1, 3), (-1, 4), (0, 2), (0, 12), (1, 3), (2, 4), (2, 12)])
def test_prover_across_forms(ctx, oracle, threads, ratio_log, group_log):
    log_size, rounds = 13, 12  # layers of 2^13 down to 4 values, every round's tree checked through the transcript
    treelet = threads.bit_length() - 1 + ratio_log
    ev = _evaluations(1 << log_size, threads + ratio_log)
    p = azk.CirclePCSFRIProver(ctx, log_size, 2, 9, rounds, schedule=dict(treelet_log=treelet, group_log=group_log, threads=threads))
    want = oracle.prove(log_size, ev, 2, 9, PUB, rounds).proof
    assert p.prove_evaluations(ev, PUB) == want
    assert p.prove_evaluations(ev, PUB) == want  # counters and transcript base as before


@pytest.mark.parametrize("log_size", range(1, 9))
def test_smallest_trees(ctx, oracle, log_size):
    """Every round down to a final layer of one value: trees of 2^k leaves, k = 8 .. 1."""
    ev = _evaluations(1 << log_size, log_size)
    assert azk.CirclePCSFRIProver(ctx, log_size, 1, 3, log_size).prove_evaluations(ev, PUB) == oracle.prove(log_size, ev, 1, 3, PUB, log_size).proof


@pytest.mark.parametrize("threads,treelet", [(128, 6), (128, 9), (256, 8), (512, 3)])
def test_64_byte_leaves_across_forms(ctx, oracle, threads, treelet):
    log_size, rounds = 12, 8
    ev_coeffs = _evaluations(1 << (log_size - 2), threads + treelet)
    b = azk.BatchProver(ctx, [log_size], [rounds], 2, 4, schedule=dict(treelet_log=treelet, threads=threads), leaf_bytes=64)
    b.upload(ev_coeffs, [0], [len(ev_coeffs)])
    b.prove(PUB)
    cm, ch, fl, _ = b.trace(0)
    full = np.zeros((1 << log_size, 4), np.uint32)
    full[: len(ev_coeffs)] = ev_coeffs
    ocm, och, ofl = oracle.commit_fold_chain_leaf64(log_size, oracle.fft_evaluate(log_size, full), 2, 4, PUB, rounds)
    assert cm == ocm and np.array_equal(ch, och) and np.array_equal(fl, ofl)


@pytest.mark.parametrize("length,stride", [(0, 1), (7, 7), (8, 8), (64, 64), (129, 131), (135, 136), (136, 136)])
@pytest.mark.parametrize("log_count", [0, 3, 4, 7, 10])
def test_raw_leaves_by_pairs(ctx, oracle, length, stride, log_count):
    """Raw leaves of every padding case, aligned or not, hashed by lane pairs."""
    n = 1 << log_count
    leaves = G.make_leaves(n, stride, length, salt=length)
    assert azk.SHA3RawLeavesMerkleCommitPlan(ctx, n, stride, length, treelet_log=7).commit(leaves) == oracle.merkle_root(leaves, n, stride, length)


@pytest.mark.parametrize("log_count", [0, 1, 3, 4, 8, 11])
def test_prehashed_digests(ctx, oracle, log_count):
    d = np.random.default_rng(log_count).integers(0, 256, 32 << log_count, dtype=np.uint8).tobytes()
    assert azk.SHA3PrehashedLeavesMerkleCommitPlan(ctx, 1 << log_count).commit(d) == oracle.merkle_root_prehashed(d)
