"""Several threads, each with a plan of its own, in calls that end in results on the
host: every thread gets its calls through (none waits until the others stop), and
every result is the one the call gives alone."""
import ctypes
import hashlib
import threading
import time

import numpy as np
import pytest
import torch

import apple_b200 as azk
from apple_b200._capi import lib
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


def test_results_larger_than_a_landing(ctx, oracle):
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
    assert sum(b.proof_sizes) > 2 << 20  # more than a landing holds
    p = azk.CirclePCSFRIProver(ctx, 16, 2, 16, 10)
    proofs = b.proofs()
    for i in (0, 7, 23):
        assert proofs[i] == p.prove_coefficients(c[i << 14:(i + 1) << 14], PUB)


def test_results_into_page_locked_memory(ctx):
    """The same proofs into page-locked and pageable memory of the caller's, through each of
    the library's downloads."""
    logs = [14] * 6
    counts = [1 << 12] * 6
    c = np.random.default_rng(4).integers(0, G.P, (sum(counts), 4), dtype=np.uint32)
    b = azk.BatchProver(ctx, logs, [8] * 6, 2, 48)
    b.upload(c, [k << 12 for k in range(6)], counts)
    b.prove(PUB * 6)
    want = b"".join(b.proofs())
    locked = torch.full((b.proof_total,), 0xA5, dtype=torch.uint8, pin_memory=True)
    pageable = np.full(b.proof_total, 0xA5, np.uint8)
    at = np.cumsum([0] + b.proof_sizes[:-1])
    for base, view in ((locked.data_ptr(), locked.numpy()), (pageable.ctypes.data, pageable)):
        assert lib().azk_batch_download_proofs(b._h, ctypes.c_void_p(base), b.proof_total) == 0
        assert view.tobytes() == want
        view[:] = 0
        outs = (ctypes.c_void_p * 6)(*[base + int(o) for o in at])
        assert lib().azk_batch_download_each(b._h, outs, (ctypes.c_uint64 * 6)(*b.proof_sizes)) == 0
        assert view.tobytes() == want
    # one result of each kind in a call
    mixed = [locked.data_ptr() + int(o) if k % 2 else pageable.ctypes.data + int(o) for k, o in enumerate(at)]
    locked.zero_()
    pageable[:] = 0
    assert lib().azk_batch_download_each(b._h, (ctypes.c_void_p * 6)(*mixed), (ctypes.c_uint64 * 6)(*b.proof_sizes)) == 0
    for k, o in enumerate(at):
        view = locked.numpy() if k % 2 else pageable
        assert view[o:o + b.proof_sizes[k]].tobytes() == want[o:o + b.proof_sizes[k]]


def test_a_thread_for_every_call(ctx):
    """Results through threads that live for one call, more of them at a time than the
    context keeps landings, small and large in turn."""
    calls = [_hash(ctx, 1), _large_codeword(ctx, 2), _prove(ctx, 3)]
    want = [call() for call in calls]
    plans = [[_hash(ctx, 1), _large_codeword(ctx, 2), _prove(ctx, 3)][k % 3] for k in range(40)]
    got = [None] * 120

    def one(i):
        got[i] = plans[i % 40]()

    for _ in range(2):
        threads = [threading.Thread(target=one, args=(i,)) for i in range(120)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert all(got[i] == want[i % 40 % 3] for i in range(120))
