"""azk_batch_download_each: one buffer per instance, each with its capacity."""
import ctypes

import numpy as np
import pytest

import apple_b200 as azk
from apple_b200._capi import lib
from tests import generators as G

pytestmark = pytest.mark.gpu


def _download(batch, buffers, capacities):
    outs = (ctypes.c_void_p * len(buffers))(*[b.ctypes.data for b in buffers])
    return lib().azk_batch_download_each(batch._h, outs, (ctypes.c_uint64 * len(buffers))(*capacities))


@pytest.mark.parametrize("short", [0, 2])
def test_a_buffer_that_is_too_small_is_refused(ctx, short):
    batch = azk.BatchProver(ctx, [8, 9, 10], [2, 3, 4], 2, 16)
    counts = [64, 128, 256]
    x = np.random.default_rng(1).integers(0, G.P, (sum(counts), 4), dtype=np.uint32)
    batch.upload(x, [0, 64, 192], counts)
    batch.prove(bytes(96))
    want = batch.proofs()
    sizes = list(batch.proof_sizes)
    buffers = [np.full(n + 8, 0xA5, np.uint8) for n in sizes]
    assert _download(batch, buffers, [n - (i == short) for i, n in enumerate(sizes)]) != 0
    assert all((b == 0xA5).all() for b in buffers)
    assert _download(batch, buffers, sizes) == 0
    assert [b[:n].tobytes() for b, n in zip(buffers, sizes)] == want
    assert all((b[n:] == 0xA5).all() for b, n in zip(buffers, sizes))
