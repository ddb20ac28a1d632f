"""Contexts with their own gas constant and reference pressure beside each other: each
keeps its own, whichever was created last, against the oracle with the same
parameters (tolerances of test_gpu_chem.py and test_gpu_chem_rhs.py)."""
import numpy as np
import pytest

import inputs
from test_gpu_chem import relerr, run_chem
from test_gpu_chem_rhs import FLOW, SPEC, TOL, grel, run_chem_rhs
from test_gpu_eb import to_dev

pytestmark = pytest.mark.gpu
PARMS = [(8.31446261815324, 101325.0), (8.0, 9.0e4), (8.6, 1.2e5)]


def test_contexts_keep_their_parameters():
    import ocfd
    from ocfd.context import default_parm
    from oracle import Oracle
    sets = []
    for Ru, Patm in PARMS:
        p, o = default_parm(), Oracle()
        p.Ru = o.parm.Ru = Ru
        p.Patm = o.parm.Patm = Patm
        sets.append((ocfd.Context(p), o))
    for ctx, o in sets:
        S, sp = inputs.chem_state(7, 6, 5, seed=91, oracle=o)
        dxinv = [1.0e4, 1.1e4, 0.9e4]
        ref, got = o.rhs_chem(S, sp, dxinv), run_chem_rhs(ctx, S, sp, (0, 0, 0), dxinv, True)
        assert grel(got[0], ref[0], FLOW) < TOL and grel(got[1], ref[1], SPEC) < TOL
        So, Ro = (np.ascontiguousarray(x.reshape(len(x), -1)) for x in (S, sp))
        Sg, Rg = run_chem(ctx, So, Ro, 1e-7)
        o.chem_advance(So, Ro, 1e-7)
        assert relerr(Sg[4], So[4]) < 1e-11
        assert np.abs(Rg - Ro).max() / np.abs(Ro).max() < 1e-11


@pytest.mark.parametrize("eb", [False, True])
def test_floor_of_negative_zero(eb):
    """A floor of -0 acts as 0 does, on cells of negative density and pressure."""
    import torch
    import ocfd
    from ocfd.context import default_parm
    n = (12, 10, 8)
    S = inputs.ideal_state(*n, seed=3)
    S[4, 7:9, 7:9, 7:9] *= 0.01
    S[0, 9, 6, 10] *= -1.0
    St, out = torch.from_numpy(S).cuda(), []
    geom = to_dev(inputs.cylinder_box(*n))
    for zero in (0.0, -0.0):
        p = default_parm()
        p.smallr = p.smallp = zero
        dS = torch.full((5,) + n[::-1], -7.0, dtype=torch.float64, device="cuda")
        a = (St, dS) + ((geom,) if eb else ()) + ((0, 0, 0), tuple(m - 1 for m in n), [12.0, 10.0, 8.0], 0)
        c = ocfd.Context(p)
        (c.rhs_eb_box if eb else c.rhs_regular_box)(*a)
        torch.cuda.synchronize()
        out.append(dS.cpu().numpy())
    assert np.array_equal(out[0], out[1], equal_nan=True)
