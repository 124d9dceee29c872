"""Hashes of messages at every byte alignment and padding case, into outputs of every
alignment, against hashlib; and raw leaves of unaligned strides against the oracle."""
import hashlib

import numpy as np
import pytest

import apple_b200 as azk
from tests import generators as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [1, 3, 7, 8, 9, 31, 32, 64, 99, 128, 131, 135, 136])
@pytest.mark.parametrize("gap,in_offset,out_stride,out_offset", [(0, 0, 32, 0), (0, 1, 32, 16), (3, 2, 40, 8), (5, 7, 33, 3), (1, 4, 48, 0)])
def test_messages_at_any_alignment(ctx, length, gap, in_offset, out_stride, out_offset):
    count, stride = 131, length + gap
    data = np.random.default_rng(1000 * length + gap).integers(0, 256, count * stride, dtype=np.uint8)
    src, dst = ctx.alloc(in_offset + count * stride), ctx.alloc(out_offset + count * out_stride)
    src.upload(data, in_offset)
    plan = azk.SHA3FixedOneBlockHashPlan(ctx, count, stride, length, output_stride=out_stride)
    plan.hash_resident(src.ptr, dst.ptr, in_offset, out_offset)
    got = np.frombuffer(dst.download(count * out_stride, out_offset), np.uint8).reshape(count, out_stride)
    for i in range(count):
        assert got[i, :32].tobytes() == hashlib.sha3_256(data[i * stride: i * stride + length].tobytes()).digest()
    assert not got[:, 32:].any()


@pytest.mark.parametrize("length,stride", [(1, 1), (9, 11), (33, 34), (131, 133), (136, 137)])
def test_unaligned_leaves(ctx, oracle, length, stride):
    leaves = G.make_leaves(2048, stride, length, salt=stride)
    want = oracle.merkle_root(leaves, 2048, stride, length)
    for treelet in (5, 11):
        assert azk.SHA3RawLeavesMerkleCommitPlan(ctx, 2048, stride, length, treelet_log=treelet).commit(leaves) == want
