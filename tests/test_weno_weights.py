"""The integer-pipe WENO-Z weights (weno_weights.cuh) on the CPU against exact
rational arithmetic, and the face value formed from them (device_physics.cuh
wenoz_face_d) against the reference's WENO-Z (Source/kernel/Reconstruction.H:
83-138) in exact arithmetic."""
import ctypes
import os
import subprocess
from fractions import Fraction as Q

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "opencfd-amr_gb300", "csrc")


@pytest.fixture(scope="module")
def weights(tmp_path_factory):
    d = tmp_path_factory.mktemp("wz")
    src, so = d / "wz.cpp", d / "wz.so"
    src.write_text('#include "weno_weights.cuh"\n'
                   'using namespace ocfd::wz;\n'
                   'extern "C" void w(const double* g, const double* e, double* c) {\n'
                   '  Weights w = weights(g[0], g[1], g[2], curvature(e[0]), curvature(e[1]), curvature(e[2]));\n'
                   '  auto over = [&](Num b, int s) { return pack(normalise(mul_hi(b.m, w.z), b.e - w.e - 61 - s)); };\n'
                   '  c[0] = over(w.b1, 0); c[1] = over(w.b2, 0); c[2] = over(w.b3, 1);\n'
                   '  c[3] = correction(w, e[0], e[1], __builtin_fma(3.0, e[1], -e[2])); }\n')
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def f(g, e):
        c = (ctypes.c_double * 4)()
        lib.w((ctypes.c_double * 3)(*g), (ctypes.c_double * 3)(*e), c)
        return list(c)
    return f


def exact_coefficients(g, e):
    D = [Q(1e-6) + Q(x) ** 2 / 4 + Q(13, 12) * Q(y) ** 2 for x, y in zip(g, e)]
    q, t = [x ** 2 for x in D], (D[0] - D[2]) ** 2
    A = [q[1] * q[2] * (q[0] + t), q[0] * q[2] * (q[1] + t), q[0] * q[1] * (q[2] + t)]
    s = A[0] + 6 * A[1] + 3 * A[2]
    # the error of tau, the difference of two indicators within 2^-55, in the weights
    d = Q(2) ** -55 * max(D[0], D[2])
    amp = max((2 * abs(D[0] - D[2]) * d + d * d) / (x + t) for x in q)
    return [A[0] / (3 * s), 2 * A[1] / s, A[2] / (2 * s)], amp


# Relative error bound.  An indicator is a sum of two squares, each truncated by less
# than 2^-55; the weights take it to at most the fourth power; tau's error is the
# indicators' and is followed exactly (amp: FP64 arithmetic has eight times as much).
# A product keeps at least 55 bits and is truncated by less than 2, so A_k and the
# sum add 0.8 units of 2^-53 each, the reciprocal and the last products less than
# 0.1, the rounding 1.
TOL = 4 * 2.0 ** -53


@pytest.mark.parametrize("lo,hi", [(-12, -6), (-3, -1), (-2, 0), (-6, 5), (-3, 22), (18, 24)])
def test_weights_exact(weights, lo, hi):
    rng = np.random.default_rng(abs(int(100 * hi)))
    for n in range(400):
        g, e = [[float(x) for x in 10.0 ** rng.uniform(lo, hi, 3) * rng.choice([-1, 1], 3)] for _ in range(2)]
        if n % 5 == 1:
            g[2], e[2] = g[0] * (1 + 2.0 ** -40 * rng.standard_normal()), -e[0]
        if n % 5 == 2:
            g[1] = g[2] = g[0]
            e[1] = e[2] = e[0]
        if n % 5 == 3:  # powers of two and their neighbours: every carry of the mantissas
            g = [float(np.nextafter(2.0 ** np.ceil(np.log2(abs(x))), rng.choice([0.0, 1e300]))) for x in g]
        if n % 5 == 4:
            g[n % 3], e[(n + 1) % 3] = 0.0, 0.0
        want, amp = exact_coefficients(g, e)
        c = weights(g, e)
        # the correction: each coefficient's error, one rounding, the alignment's 2^-57
        terms = [want[0] * Q(e[0]), want[1] * Q(e[1]), 3 * want[2] * Q(e[1]), -want[2] * Q(e[2])]
        assert abs(Q(c[3]) - sum(terms)) <= (Q(TOL) + 2 * amp) * sum(abs(t) for t in terms)
        for got, w in zip(c, want):
            if w < Q(2) ** -1000:
                assert 0 <= got <= 2.0 ** -999
            else:
                assert abs(Q(got) - w) <= (Q(TOL) + 2 * amp) * w


def test_weights_flat(weights):
    # zero and denormal differences: the linear weights
    for x in (0.0, 5e-324, 1e-310, 1e-200):
        c = weights([x, -x, 0.0], [x, 0.0, -x])
        assert np.allclose(c[:3], [1 / 30, 6 / 30, 3 / 60], rtol=2 ** -52, atol=0)
    assert weights([0.0] * 3, [0.0, -0.0, 0.0])[3] == 0.0 and weights([1.0, 2.0, -3.0], [0.0] * 3)[3] == 0.0


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_correction_not_finite(weights, bad):
    for k in range(3):
        e = [1.0, -2.0, 0.5]
        e[k] = bad
        assert np.isnan(weights([1.0, 1.0, bad], e)[3])


def face(weights, V):
    d = [V[i + 1] - V[i] for i in range(4)]
    e = [d[i + 1] - d[i] for i in range(3)]
    c = weights([2 * d[1] + e[0], d[1] + d[2], 2 * d[2] - e[2]], e)
    return (V[2] + 0.5 * d[1]) + c[3]


def face_exact(V):
    a, b, c, d, e = [Q(float(x)) for x in V]
    be = [Q(13, 12) * (a - 2 * b + c) ** 2 + Q(1, 4) * (a - 4 * b + 3 * c) ** 2,
          Q(13, 12) * (b - 2 * c + d) ** 2 + Q(1, 4) * (b - d) ** 2,
          Q(13, 12) * (c - 2 * d + e) ** 2 + Q(1, 4) * (3 * c - 4 * d + e) ** 2]
    t, eps = abs(be[0] - be[2]), Q(1e-6)
    w = [g * (1 + (t / (eps + x)) ** 2) for g, x in zip((1, 6, 3), be)]
    v = [2 * a - 7 * b + 11 * c, -b + 5 * c + 2 * d, 2 * c + 5 * d - e]
    return sum(x * y for x, y in zip(w, v)) / (6 * sum(w))


@pytest.mark.parametrize("scale", [1e-8, 1e-3, 1.0, 1e4, 1e8])
def test_face_value(weights, scale):
    rng = np.random.default_rng(3)
    for n in range(200):
        if n % 3 == 0:
            V = np.sin(rng.uniform(0, 6) + np.arange(5) * rng.uniform(0.01, 0.5)) + 1.5
        elif n % 3 == 1:
            V = rng.standard_normal(5)
        else:
            V = np.where(np.arange(5) < rng.integers(1, 5), 1.0, 10.0 ** rng.uniform(-3, 3)) * (1 + 1e-3 * rng.random(5))
        V = [float(x) for x in scale * V]
        # indicators within 10 roundings, which the weights double; candidates of at most
        # 7 max |V| with the weights' errors; four roundings of the sum
        assert abs(Q(face(weights, V)) - face_exact(V)) <= Q(2.0 ** -53 * 200 * max(abs(x) for x in V))


@pytest.mark.parametrize("mid", [0.0, 1e-3, 1.0, 30.0])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("p", range(3, 16))
def test_plateau_between_equal_jumps(weights, p, sign, mid):
    # tau is exactly zero, the middle indicator far below the outer two: the linear
    # weights, whatever the indicators' ratio
    a = 10.0 ** p
    g, e = [a, mid, sign * a], [a, 0.0, -sign * a]
    c = weights(g, e)
    for got, w in zip(c, (Q(1, 30), Q(1, 5), Q(1, 20))):
        assert abs(Q(got) - w) <= Q(TOL) * w
    V = [1.0 + a, 1.0, 1.0, 1.0, 1.0 + sign * a]
    # the values' differences are exact; three terms of at most a / 5, each within TOL,
    # and two roundings of the sum
    assert abs(Q(face(weights, V)) - face_exact(V)) <= (Q(TOL) + Q(2.0 ** -52)) * Q(a)
