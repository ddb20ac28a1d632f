"""The fused chemistry substep at the edges of its ranges against the oracle:
temperatures on both sides of the fits' 1000 K joint and beyond their 250-3500 K
range, cells without radicals (exactly zero concentrations), large steps, and cell
counts around one block."""
import numpy as np
import pytest

from test_gpu_chem import ctx, relerr, run_chem  # noqa: F401

pytestmark = pytest.mark.gpu


def states(oracle, n, T, radicals, seed):
    rng = np.random.default_rng(seed)
    S, R = np.zeros((5, n)), np.zeros((9, n))
    for c in range(n):
        X = np.zeros(9)
        X[0], X[1], X[2] = rng.uniform(0.1, 0.3), rng.uniform(0.05, 0.2), rng.uniform(0.0, 0.2)
        if radicals:
            X[3:8] = rng.uniform(0.0, 5e-3, 5)
        X[8] = 1.0 - X.sum()
        t = T[c % len(T)]
        Y = oracle.ckxty(X)
        rho = oracle.ckrhoy(101325.0, max(t, 250.0), Y)
        u = 100.0 * rng.standard_normal(3)
        R[:, c] = rho * Y
        S[0, c], S[1:4, c] = rho, rho * u
        S[4, c] = oracle.ckubms(t, R[:, c]) + 0.5 * rho * (u * u).sum()
    return S, R


# the tolerance of test_gpu_chem.py: exponentials and logarithms a few ulps off the host's,
# amplified by activation temperatures of up to 5e4 K
@pytest.mark.parametrize("n,radicals,dt", [(1, True, 1e-8), (127, True, 1e-7), (129, False, 1e-8), (300, True, 1e-5)])
@pytest.mark.parametrize("T", [(252.0, 400.0, 700.0), (999.9, 1000.1, 1003.0), (180.0, 2400.0, 3499.0, 3800.0)])
def test_chem_edges(ctx, oracle, n, radicals, dt, T):  # noqa: F811
    S, R = states(oracle, n, T, radicals, seed=n)
    So, Ro = S.copy(), R.copy()
    oracle.chem_advance(So, Ro, dt)
    Sg, Rg = run_chem(ctx, S, R, dt)
    assert np.isfinite(Sg).all() and np.isfinite(Rg).all()
    assert relerr(Sg[4], So[4]) < 1e-11
    assert np.abs(Rg - Ro).max() / np.abs(Ro).max() < 1e-11
    assert np.array_equal(Rg[8], R[8])  # N2 takes part in no reaction
