"""GPU parity of the witness transform's fast convolutions with the CPU oracle: sizes
around every change of path (direct sum, one-CTA convolutions, one and more strided
stages, one and more line-basis launches), QM31 and lifted columns, uneven lengths."""
import numpy as np
import pytest

import apple_b200 as azk
from tests import generators as G

pytestmark = pytest.mark.gpu


def _column(rng, n, lifted):
    c = rng.integers(0, G.P, size=(n, 4), dtype=np.uint32)
    if lifted:
        c[:, 1:] = 0
    return c


@pytest.mark.parametrize("lifted", [False, True])
@pytest.mark.parametrize("log_size,nx,ny", [(12, 1025, 2048), (13, 1, 2049), (13, 4096, 0), (14, 5000, 8192), (15, 16384, 16383), (16, 20000, 1),
                                            (18, 3, 2)])
def test_convolution_sizes_match_oracle(ctx, oracle, log_size, nx, ny, lifted):
    rng = np.random.default_rng(log_size * 1000 + nx)
    x, y = _column(rng, nx, lifted), _column(rng, ny, lifted)
    got = azk.CircleWitnessToFFTBasisPlan(ctx, log_size).execute(x, y)
    assert np.array_equal(got, oracle.fft_basis_coefficients(log_size, x, y))


def _convert_by_evaluation(ctx, log_size, x, y):
    """The codeword of the converted coefficients at the domain's points, and the
    polynomial there by Horner's rule in 64-bit integers (base-field columns)."""
    code = azk.CircleCodewordPlan(ctx, log_size).execute(x, y)
    pts = azk.circle_domain_points(ctx, log_size).astype(np.uint64)
    at = np.random.default_rng(log_size).integers(0, 1 << log_size, 40)
    px, py = pts[at, 0], pts[at, 1]
    p = np.uint64(G.P)
    vx, vy = np.zeros(len(at), np.uint64), np.zeros(len(at), np.uint64)
    for c in x[::-1, 0]:
        vx = (vx * px + np.uint64(c)) % p
    for c in y[::-1, 0]:
        vy = (vy * px + np.uint64(c)) % p
    return code[at], (vx + py * vy) % p


@pytest.mark.parametrize("log_size,nx,ny", [(18, 1 << 17, 100001), (20, 1 << 18, 1 << 17)])
def test_long_columns_evaluate_right(ctx, log_size, nx, ny):
    rng = np.random.default_rng(log_size)
    code, want = _convert_by_evaluation(ctx, log_size, _column(rng, nx, True), _column(rng, ny, True))
    assert np.array_equal(code[:, 0], want.astype(np.uint32)) and not code[:, 1:].any()


def test_lifted_and_general_agree_at_full_size(ctx):
    """2^22 domain: the two-column transform of base-field columns is the general
    one's base limb (linearity in each limb)."""
    rng = np.random.default_rng(22)
    n = 1 << 19
    x, y = _column(rng, n, False), _column(rng, n, False)
    plan = azk.CircleWitnessToFFTBasisPlan(ctx, 22)
    full = plan.execute(x, y)
    for limb in (0, 3):
        lx, ly = np.zeros_like(x), np.zeros_like(y)
        lx[:, 0], ly[:, 0] = x[:, limb], y[:, limb]
        got = plan.execute(lx, ly)
        assert np.array_equal(got[:, 0], full[:, limb]) and not got[:, 1:].any()


def test_one_plan_serves_columns_of_every_length(ctx, oracle):
    """Workspace grown and reused: long, short, long columns through one plan."""
    rng = np.random.default_rng(5)
    plan = azk.CircleWitnessToFFTBasisPlan(ctx, 14)
    for n in (3000, 8192, 5, 1500, 8192, 2049):
        x, y = _column(rng, n, n == 1500), _column(rng, max(1, n - 7), n == 1500)
        assert np.array_equal(plan.execute(x, y), oracle.fft_basis_coefficients(14, x, y))
