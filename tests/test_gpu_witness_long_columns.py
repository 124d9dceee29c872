"""The longest witness columns (up to 2^21 coefficients, a 2^22 domain): the codeword
at sampled domain points against Horner's rule in 64-bit integers.  The points are base-field, so the limbs of a
general column are four independent polynomials there."""
import numpy as np
import pytest

import apple_b200 as azk
from tests import generators as G

pytestmark = pytest.mark.gpu

_P = np.uint64(G.P)
POINTS = 24


def _horner(column, px):
    """Every limb of the column at the points px: (points, 4)."""
    v = np.zeros((len(px), 4), np.uint64)
    # blocks of coefficients by powers of px, then Horner's rule over the blocks
    block = 1 << 11
    powers = np.ones((len(px), block), np.uint64)
    for k in range(1, block):
        powers[:, k] = powers[:, k - 1] * px % _P
    step = powers[:, -1] * px % _P
    c = column.astype(np.uint64)
    for at in range((len(c) - 1) // block * block, -1, -block):
        part = c[at:at + block]
        s = np.zeros_like(v)
        for limb in range(4):
            s[:, limb] = (powers[:, :len(part)] * part[None, :, limb] % _P).sum(axis=1) % _P
        v = (v * step[:, None] + s) % _P
    return v


@pytest.mark.parametrize("lifted", [False, True])
@pytest.mark.parametrize("log_size,nx,ny", [(20, 1 << 19, (1 << 18) + 1), (21, 1 << 20, 77), (22, 1 << 20, 1 << 20), (22, (1 << 20) + 1, 1 << 19), (22, 1 << 21, 1 << 21)])
def test_long_columns_evaluate_right(ctx, log_size, nx, ny, lifted):
    rng = np.random.default_rng(log_size + nx)
    x, y = (rng.integers(0, G.P, size=(n, 4), dtype=np.uint32) for n in (nx, ny))
    if lifted:
        x[:, 1:] = 0
        y[:, 1:] = 0
    code = azk.CircleCodewordPlan(ctx, log_size).execute(x, y)
    pts = azk.circle_domain_points(ctx, log_size).astype(np.uint64)
    at = rng.integers(0, 1 << log_size, POINTS)
    px, py = pts[at, 0], pts[at, 1]
    want = (_horner(x, px) + py[:, None] * _horner(y, px)) % _P
    assert np.array_equal(code[at], want.astype(np.uint32))
