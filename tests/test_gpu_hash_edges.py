"""Hash batches whose first and last message share a warp, a CTA or neither, at every
byte alignment of the buffer's ends, with bytes around the batch that must not enter a
digest."""
import hashlib

import numpy as np
import pytest

import apple_b200 as azk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [64, 256])
@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 64, 65, 257])
@pytest.mark.parametrize("length,stride", [(1, 1), (2, 5), (6, 7), (63, 65), (97, 99), (131, 131), (135, 137), (136, 139)])
def test_first_and_last_message(ctx, count, length, stride, threads):
    rng = np.random.default_rng(1000 * count + length)
    plan = azk.SHA3FixedOneBlockHashPlan(ctx, count, stride, length, threads=threads)
    dst = ctx.alloc(32 * count)
    for offset in range(4):
        data = rng.integers(0, 256, offset + count * stride + 8, dtype=np.uint8)
        src = ctx.alloc(len(data))
        src.upload(data)
        plan.hash_resident(src.ptr, dst.ptr, offset, 0)
        got = dst.download(32 * count)
        for i in {0, count // 2, count - 1}:
            at = offset + i * stride
            assert got[32 * i:32 * i + 32] == hashlib.sha3_256(data[at:at + length].tobytes()).digest(), (offset, i)
