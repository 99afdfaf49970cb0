"""rf_smooth_F and rf_check_F against numpy in 64 bits: matrices whose rows fit shared
memory, those whose rows do not, row counts around the number of SMs, rows without
rays, surfaces without area."""
import numpy as np
import pytest

from rayfactorcl_gb300.tracer import Tracer

pytestmark = pytest.mark.gpu


def exchange(n, seed):
    """A closed enclosure's F with Monte Carlo noise: a positive symmetric kernel that
    couples near surfaces more, scaled to its areas."""
    rng = np.random.default_rng(seed)
    z = np.sort(rng.uniform(0, 1, n))
    A = rng.uniform(0.5, 1.5, n)
    K = np.exp(-4.0 * np.abs(z[:, None] - z[None, :])) * A[:, None] * A[None, :]
    x = np.ones(n)
    for _ in range(200):
        x = np.sqrt(x * A / (K @ x))
    F = x[:, None] * K * x[None, :] / A[:, None]
    return F * (1.0 + 0.02 * rng.standard_normal((n, n))), A


def smooth(F, A, closed):
    Fz = np.nan_to_num(F, nan=0.0)
    G = 0.5 * (A[:, None] * Fz + (A[:, None] * Fz).T)
    x = np.ones(len(A))
    if closed:
        for it in range(2000):
            s = G @ x
            live = (s > 0) & (A > 0)
            err = np.max(np.abs(x * s / np.where(A > 0, A, 1) - 1)[live], initial=0.0)
            x = np.where(live, np.sqrt(x * A / np.where(live, s, 1)), x)
            if it % 8 == 7 and err <= 1e-13:
                break
    with np.errstate(divide="ignore", invalid="ignore"):
        return np.where(A[:, None] > 0, x[:, None] * G * x[None, :] / A[:, None], 0.0)


@pytest.mark.parametrize("closed", [True, False])
@pytest.mark.parametrize("n", [1, 2, 31, 152, 153, 300, 2100])
def test_smoothing(built_lib, n, closed):
    F, A = exchange(n, n)
    if n >= 31:
        F[3] = np.nan     # a row without rays
        A[5] = 0.0        # a surface without area
    with Tracer() as t:
        got, it, res = t.smooth_F(F, A, closed=closed)
        again, _, _ = t.smooth_F(F, A, closed=closed)
    ref = smooth(F, A, closed)
    # sums of n products in another order: n 2^-53 relative, a few times over for the
    # square root's argument and the two scalings
    tol = 8 * (n + 8) * 2.0 ** -53
    assert np.max(np.abs(got - ref)) <= tol * np.max(np.abs(ref)) + 4e-13 * np.max(np.abs(ref))
    assert np.array_equal(got, again)
    if closed:
        assert it % 8 == 0 and (res <= 1e-13 or it == 2000)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 300])
def test_check(built_lib, n):
    F, A = exchange(n, n + 1)
    if n > 2:
        F[1, 2] = 0.0
    with Tracer() as t:
        s, r = t.check_F(F, A)
        s0, r0 = t.check_F(F)
    AF = A[:, None] * F
    both = (F > 0) & (F.T > 0)
    ref_r = np.max(np.where(both, np.abs(AF - AF.T) / np.maximum(AF, AF.T), 0.0))
    ref_s = np.max(np.abs(F.sum(axis=1) - 1))
    assert abs(s - ref_s) <= 4 * n * 2.0 ** -53 * np.max(np.sum(np.abs(F), axis=1)) + 2.0 ** -52
    assert abs(r - ref_r) <= 8 * 2.0 ** -53 and s0 == s and r0 == 0.0
