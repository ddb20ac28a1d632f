"""The FP64 Steger-Warming split gives un's side its outer eigenvalue and places the
inner one by its sign: streams at rest, sub- and supersonic and exactly sonic (the
inner eigenvalue is zero) of either sign along each direction, the first cells of
every line undisturbed (flat lines keep their value at each face), against the
oracle.  Tolerance: that of the other parity tests of the right-hand side, 1e-12 of
the largest value, fluxes and divergence by group (a stream along x leaves the
other momenta at rounding size)."""
import numpy as np
import pytest

import inputs

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("mach", [0.0, -0.0, 0.4, -0.4, 1.0, -1.0, 3.0, -3.0])
@pytest.mark.parametrize("dim", [0, 1, 2])
def test_split_sides(oracle, dim, mach):
    import torch
    import ocfd
    n, g = (20, 17, 18), 1.4
    sh = inputs.grown(1, *n)[1:]
    rng = np.random.default_rng(7)
    part = np.arange(sh[2 - dim]) >= sh[2 - dim] // 2
    part = part.reshape([-1 if a == 2 - dim else 1 for a in range(3)])
    amp = 0.2 * part * (np.arange(sh[2 - dim]) % 4 != 0).reshape(part.shape)
    rho, p = 1.4 * (1.0 + amp * rng.random(sh)), 1.0 + amp * rng.random(sh)   # c = 1 where undisturbed
    u = np.zeros((3,) + sh)
    u[dim] = mach
    u[(dim + 1) % 3] = -0.3 * amp
    S = np.concatenate([rho[None], rho * u, (p / (g - 1) + 0.5 * rho * (u * u).sum(0))[None]])
    dxinv = [20.0, 17.0, 18.0]
    ref, rf = oracle.rhs_regular(S, dxinv)
    dS = torch.full((5,) + n[::-1], float("nan"), dtype=torch.float64, device="cuda")
    fl = [torch.full((5,) + tuple(n[d] + (d == k) for d in (2, 1, 0)), float("nan"), dtype=torch.float64,
                     device="cuda") for k in range(3)]
    ocfd.Context().rhs_regular_box(torch.from_numpy(S).cuda(), dS, (0, 0, 0), tuple(m - 1 for m in n), dxinv, 0, flux=fl)
    torch.cuda.synchronize()
    for got, want in [(dS, ref)] + list(zip(fl, rf)):
        got = got.cpu().numpy()
        for grp in ((0,), (1, 2, 3), (4,)):
            grp = list(grp)
            assert np.abs(got[grp] - want[grp]).max() <= TOL * max(np.abs(want[grp]).max(), 1e-300), grp
