"""The chemistry kernels' own functions: the one-step reciprocal and the table-driven
exponential against wider arithmetic and at the ends of their ranges, and the
temperature inversion where rounding decides on its last Newton step."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def probe(x):
    import torch
    import ocfd
    from ocfd._abi import declare
    from ocfd.context import _stream_ptr
    ocfd.load()
    declare("ocfd_check_chem_math_f64", ctypes.c_int, [ctypes.c_void_p] * 4 + [ctypes.c_int64, ctypes.c_void_p])
    xt = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    out = [torch.empty_like(xt) for _ in range(3)]
    ocfd.check(ocfd.load().ocfd_check_chem_math_f64(xt.data_ptr(), *[o.data_ptr() for o in out], x.size, _stream_ptr(None)))
    torch.cuda.synchronize()
    return [o.cpu().numpy() for o in out]


def ulps(got, want):
    """error of doubles in units of the last place of `want` (long double, normal)"""
    return np.abs((got.astype(np.longdouble) - want) / np.spacing(np.abs(want).astype(np.float64))).astype(np.float64)


def test_rcp_cubic():
    rng = np.random.default_rng(8)
    m = np.concatenate([rng.uniform(1.0, 2.0, 200000), 1.0 + np.arange(64) * 2.0 ** -52, 2.0 - np.arange(1, 64) * 2.0 ** -52])
    x = m * 2.0 ** rng.integers(-1000, 1000, m.size) * rng.choice([-1.0, 1.0], m.size)
    # one rounding, and 2^-69 / 2^-53 of a seed within 2^-23
    assert ulps(probe(x)[0], 1 / x.astype(np.longdouble)).max() <= 0.51
    # beyond: no value where 1 / x is infinite or zero
    assert not np.isfinite(probe(np.array([0.0, -0.0, np.inf, -np.inf, np.nan]))[0]).any()


def test_exp_tab():
    rng = np.random.default_rng(9)
    step = np.log(2.0) / 128
    x = np.concatenate([rng.uniform(-708.0, 708.0, 300000), rng.uniform(-2.0, 2.0, 100000), rng.normal(0, 1e-6, 1000),
                        (np.arange(-256, 257)[:, None] * step + np.array([-0.5, -0.49, -1e-3, 0.0, 1e-3, 0.49, 0.5]) * step).ravel(),
                        [0.0, -0.0, 1e-300, 708.0, -708.0, np.nextafter(708.0, 0), np.nextafter(-708.0, 0),
                         np.nextafter(708.0, 800), np.nextafter(-708.0, -800)]])
    assert set((np.rint(x / step).astype(np.int64) & 127).tolist()) == set(range(128))
    assert ulps(probe(x)[1], np.exp(x.astype(np.longdouble))).max() <= 0.52
    # outside, and not finite: CUDA's own
    y = np.array([708.1, 709.7, 710.0, 1e4, np.inf, -708.1, -720.0, -745.0, -746.0, -1e300, -np.inf, np.nan])
    got, cuda = probe(y)[1:]
    assert np.array_equal(got, cuda, equal_nan=True)
    assert got[4] == np.inf and got[10] == 0.0 and np.isnan(got[11])


def newton_steps(o, e, r, n):
    p, mw, A0 = o.parm, o.parm.mw, o.parm.A0
    t = e / sum(A0[k] * p.Ru / mw[k] * r[k] for k in range(9))
    rp = r.ctypes.data_as(ctypes.c_void_p)
    out = []
    for _ in range(n):
        dt = (e - o.ckubms(t, r)) / o.lib.ocfdo_ckcvbs(o.pp, t, rp)
        out.append(abs(dt))
        t += max(-100.0, min(100.0, dt))
    return out


def close_steps(o, offsets):
    """(e, partial densities) whose Newton step number k is 1e-7 K plus an offset"""
    rng = np.random.default_rng(12)
    E, R = [], []
    for _ in range(4):
        X = rng.uniform(0.0, [0.3, 0.2, 0.2, 0.01, 0.01, 0.01, 0.01, 0.01, 0.0])
        X[8] = 1.0 - X.sum()
        Y = o.ckxty(X)
        r = o.ckrhoy(101325.0, 1000.0, Y) * Y
        grid = [o.ckubms(T, r) for T in np.linspace(300.0, 2900.0, 60)]
        st = [newton_steps(o, e, r, 14) for e in grid]
        for i in range(len(grid) - 1):
            for k in range(14):
                if (st[i][k] - 1e-7) * (st[i + 1][k] - 1e-7) >= 0 or max(st[i][k], st[i + 1][k]) > 1e-4:
                    continue
                for off in offsets:
                    a, b = grid[i], grid[i + 1]
                    up = st[i + 1][k] > st[i][k]
                    for _ in range(60):
                        mid = 0.5 * (a + b)
                        if (newton_steps(o, mid, r, k + 1)[k] > 1e-7 + off) == up:
                            b = mid
                        else:
                            a = mid
                    if abs(newton_steps(o, b, r, k + 1)[k] - 1e-7 - off) < 1e-12:
                        E.append(b)
                        R.append(r)
    return np.array(E), np.array(R).T


def test_last_newton_step(oracle):
    """A step is dropped below 1e-7 K: GPU and oracle decide alike where the step lies
    within rounding's reach of the tolerance, inside the window that is run again in the
    reference's order and on both sides of its ends."""
    import torch
    import ocfd
    from ocfd import surrogate
    E, R = close_steps(oracle, [s * d for d in (4e-12, 8e-12, 1.3e-11, 3e-11) for s in (-1, 1)])
    assert E.size >= 16
    U = np.zeros((14, E.size))
    U[0], U[4], U[5:] = R.sum(0), E, R
    T = surrogate.cells_props(ocfd.Context(), torch.from_numpy(U).cuda())[0].cpu().numpy()
    want = np.array([oracle.get_t_given_ey(e, r) for e, r in zip(E, R.T)])
    assert np.abs(T - want).max() < 1e-9  # a step more or less is 1e-7 K
