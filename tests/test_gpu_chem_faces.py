"""Multispecies face tiles (8 lines x 24 faces) at their edges - a single cell, lines
and faces one short of, at and one past a tile - against the oracle, with the
tolerance of test_gpu_chem_rhs.py."""
import numpy as np
import pytest

import inputs
from test_gpu_chem_rhs import FLOW, SPEC, TOL, ctx, grel, run_chem_rhs  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("visc", [False, True])
@pytest.mark.parametrize("shape", [(1, 1, 1), (22, 3, 3), (23, 7, 1), (24, 2, 4), (3, 25, 2), (2, 1, 48)])
def test_chem_face_tile_edges(ctx, oracle, visc, shape):  # noqa: F811
    S, sp = inputs.chem_state(*shape, seed=sum(shape), oracle=oracle)
    dxinv = [1.0e4, 1.1e4, 0.9e4]
    ref = oracle.rhs_chem(S, sp, dxinv, do_visc=visc)
    got = run_chem_rhs(ctx, S, sp, (5, -2, 1), dxinv, visc)
    assert grel(got[0], ref[0], FLOW) < TOL and grel(got[1], ref[1], SPEC) < TOL
    for d in range(3):
        assert np.isfinite(got[2][d]).all() and np.isfinite(got[3][d]).all()
        assert grel(got[2][d], ref[2][d], FLOW) < TOL and grel(got[3][d], ref[3][d], SPEC) < TOL
