"""Several threads, each with a plan of its own, in calls that end in results on the
host: every thread gets its calls through (none waits until the others stop), and
every result is the one the call gives alone."""
import hashlib
import threading
import time

import numpy as np
import pytest

import apple_b200 as azk
from tests import generators as G

pytestmark = pytest.mark.gpu
THREADS, SECONDS = 12, 0.6
PUB = bytes(range(32))


def _prove(ctx, seed):
    p = azk.CirclePCSFRIProver(ctx, 12, 2, 32, 6)
    x = np.random.default_rng(seed).integers(0, G.P, (1 << 10, 4), dtype=np.uint32)
    return lambda: p.prove_coefficients(x, PUB)


def _prove_evaluations(ctx, seed):
    p = azk.CirclePCSFRIProver(ctx, 10, 2, 16, 4)
    x = np.random.default_rng(seed).integers(0, G.P, (1 << 10, 4), dtype=np.uint32)
    return lambda: p.prove_evaluations(x, PUB)


def _hash(ctx, seed):
    p = azk.SHA3FixedOneBlockHashPlan(ctx, 4096, 32, 32)
    m = np.random.default_rng(seed).integers(0, 256, 4096 * 32, dtype=np.uint8)
    return lambda: p.hash(m)


def _commit(ctx, seed):
    p = azk.SHA3PrehashedLeavesMerkleCommitPlan(ctx, 1 << 10)
    d = np.random.default_rng(seed).integers(0, 256, 1 << 15, dtype=np.uint8).tobytes()
    return lambda: p.commit(d)


def _codeword(ctx, seed):
    p = azk.CircleCodewordPlan(ctx, 12)
    x = np.random.default_rng(seed).integers(0, G.P, (1 << 12, 4), dtype=np.uint32)
    return lambda: p.execute_coefficients(x).tobytes()


def _large_codeword(ctx, seed):
    p = azk.CircleCodewordPlan(ctx, 18)
    x = np.random.default_rng(seed).integers(0, G.P, (1 << 18, 4), dtype=np.uint32)
    return lambda: p.execute_coefficients(x)[::64].tobytes()


@pytest.mark.parametrize("make", [_prove, _prove_evaluations, _hash, _commit, _codeword, _large_codeword])
def test_every_thread_gets_its_calls_through(ctx, make):
    calls = [make(ctx, seed) for seed in range(THREADS)]
    want = [hashlib.sha256(call()).digest() for call in calls]
    done, wrong = [0] * THREADS, []
    stop = time.monotonic() + SECONDS

    def work(i):
        while time.monotonic() < stop:
            if hashlib.sha256(calls[i]()).digest() != want[i]:
                wrong.append(i)
            done[i] += 1

    threads = [threading.Thread(target=work, args=(i,)) for i in range(THREADS)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    assert 8 * min(done) >= max(done), done


def test_results_larger_than_a_threads_landing(ctx, oracle):
    """Results that cross in pieces (4 MB of digests, a 4 MB codeword, batches of proofs whose
    sizes are no multiple of a piece), small and large ones from one thread in turn."""
    rng = np.random.default_rng(3)
    for count in (1 << 10, 1 << 17, 3):
        m = rng.integers(0, 256, (count, 32), dtype=np.uint8)
        got = np.frombuffer(azk.SHA3FixedOneBlockHashPlan(ctx, count, 32, 32).hash(m), np.uint8).reshape(count, 32)
        for i in sorted({0, count // 2, count - 1}):
            assert got[i].tobytes() == hashlib.sha3_256(m[i].tobytes()).digest()
    x = rng.integers(0, G.P, (1 << 18, 4), dtype=np.uint32)
    assert np.array_equal(azk.CircleCodewordPlan(ctx, 18).execute_coefficients(x), oracle.fft_evaluate(18, x))
    logs = [16] * 24
    counts = [(1 << lg) >> 2 for lg in logs]
    c = rng.integers(0, G.P, (sum(counts), 4), dtype=np.uint32)
    b = azk.BatchProver(ctx, logs, [10] * len(logs), 2, 16)
    b.upload(c, list(np.cumsum([0] + counts[:-1])), counts)
    b.prove(PUB * len(logs))
    assert sum(b.proof_sizes) > 2 << 20  # more than a thread's landing
    p = azk.CirclePCSFRIProver(ctx, 16, 2, 16, 10)
    proofs = b.proofs()
    for i in (0, 7, 23):
        assert proofs[i] == p.prove_coefficients(c[i << 14:(i + 1) << 14], PUB)
