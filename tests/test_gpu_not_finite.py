"""One cell that is not a number (or infinite) makes the divergence not finite in every
cell where the oracle's is not: neither side of the split, the WENO-Z weights nor the
flat-line test hides it, in streams along either sign of each direction, at rest, sub-
and supersonic."""
import numpy as np
import pytest

import inputs

pytestmark = pytest.mark.gpu
N = (16, 13, 12)


def stream(dim, mach, seed=3):
    sh = inputs.grown(1, *N)[1:]
    rng = np.random.default_rng(seed)
    rho, p = 1.4 + 0.1 * rng.random(sh), 1.0 + 0.1 * rng.random(sh)
    u = 0.05 * rng.standard_normal((3,) + sh)
    u[dim] += mach
    return np.concatenate([rho[None], rho * u, (p / 0.4 + 0.5 * rho * (u * u).sum(0))[None]])


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("comp", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("mach", [0.0, 0.5, 3.0, -3.0])
@pytest.mark.parametrize("dim", [0, 1, 2])
def test_bad_cell_shows(oracle, dim, mach, comp, bad):
    import torch
    import ocfd
    S = stream(dim, mach)
    S[comp, 4 + 6, 4 + 6, 4 + 7] = bad
    dxinv = [16.0, 13.0, 12.0]
    with np.errstate(all="ignore"):
        ref, _ = oracle.rhs_regular(S, dxinv)
    dS = torch.zeros((5,) + N[::-1], dtype=torch.float64, device="cuda")
    ocfd.Context().rhs_regular_box(torch.from_numpy(S).cuda(), dS, (0, 0, 0), tuple(m - 1 for m in N), dxinv, 0)
    torch.cuda.synchronize()
    want = ~np.isfinite(ref).all(0)
    got = ~np.isfinite(dS.cpu().numpy()).all(0)
    assert (got | ~want).all(), (int(want.sum()), int((want & ~got).sum()))


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("comp", [0, 2, 4, 5, 13])
@pytest.mark.parametrize("speed", [0.0, 3000.0, -3000.0])
@pytest.mark.parametrize("dim", [0, 1, 2])
def test_bad_cell_shows_multispecies(oracle, dim, speed, comp, bad):
    import torch
    import ocfd
    n = (9, 8, 7)
    S, sp = inputs.chem_state(*n, seed=6, oracle=oracle, vel=20.0)
    S[4] += speed * S[1 + dim] + 0.5 * S[0] * speed * speed
    S[1 + dim] += S[0] * speed
    (S if comp < 5 else sp)[comp if comp < 5 else comp - 5, 4 + 3, 4 + 4, 4 + 4] = bad
    dxinv = [1.0e4, 1.1e4, 0.9e4]
    with np.errstate(all="ignore"):
        ref = oracle.rhs_chem(S, sp, dxinv, do_visc=False)
    got = [torch.zeros((k,) + n[::-1], dtype=torch.float64, device="cuda") for k in (5, 9)]
    ocfd.Context().rhs_chem_box(torch.from_numpy(S).cuda(), torch.from_numpy(sp).cuda(), *got, (0, 0, 0),
                                tuple(m - 1 for m in n), dxinv, 0)
    torch.cuda.synchronize()
    want = ~np.isfinite(np.concatenate(ref[:2])).all(0)
    have = ~np.isfinite(torch.cat(got).cpu().numpy()).all(0)
    assert (have | ~want).all(), (int(want.sum()), int((want & ~have).sum()))
