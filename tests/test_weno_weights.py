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
                   'extern "C" void w(const double* D, double* c) '
                   '{ ocfd::wz::weights(D[0], D[1], D[2], D[3], c[0], c[1], c[2]); }\n')
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def f(D1, D2, D3, tau):
        a, c = (ctypes.c_double * 4)(D1, D2, D3, tau), (ctypes.c_double * 3)()
        lib.w(a, c)
        return list(c)
    return f


def exact_coefficients(D, tau):
    q, t = [Q(x) ** 2 for x in D], Q(tau) ** 2
    A = [q[1] * q[2] * (q[0] + t), q[0] * q[2] * (q[1] + t), q[0] * q[1] * (q[2] + t)]
    s = A[0] + 6 * A[1] + 3 * A[2]
    return [A[0] / (3 * s), 2 * A[1] / s, A[2] / (2 * s)]


# Relative error bound, in units of 2^-53: a product of two numbers below 2^63 keeps
# at least 55 bits and is truncated by less than 2, so A_k and the sum are each
# within 0.8; the reciprocal and the last products add less than 0.1; the rounding 1.
TOL = 3 * 2.0 ** -53


@pytest.mark.parametrize("lo,hi", [(-6, -5.99), (-6, 0), (-6, 10), (-3, 45), (40, 50)])
def test_weights_exact(weights, lo, hi):
    rng = np.random.default_rng(abs(int(100 * hi)))
    for n in range(400):
        D = [max(1e-6, float(x)) for x in 10.0 ** rng.uniform(lo, hi, 3)]
        if n % 5 == 1:
            D[2] = D[0] * (1 + 2.0 ** -40 * rng.standard_normal())
        if n % 5 == 2:
            D[1] = D[2] = D[0]
        if n % 5 == 3:  # powers of two and their neighbours: every carry of the mantissas
            D = [float(np.nextafter(2.0 ** np.ceil(np.log2(x)), rng.choice([0.0, 1e300]))) for x in D]
            D = [max(1e-6, x) for x in D]
        tau = abs(D[0] - D[2])
        for got, want in zip(weights(*D, tau), exact_coefficients(D, tau)):
            if want > Q(2) ** -1000:
                assert abs(Q(got) - want) <= Q(TOL) * want
            else:
                assert 0 <= got <= 2.0 ** -999


def test_weights_smooth(weights):
    # tau = 0 and denormal tau: the linear weights
    for tau in (0.0, 5e-324, 1e-310):
        c = weights(1e-6, 1e-6, 1e-6, tau)
        assert np.allclose(c, [1 / 30, 6 / 30, 3 / 60], rtol=2 ** -52, atol=0)


def face(weights, V):
    d = [V[i + 1] - V[i] for i in range(4)]
    e = [d[i + 1] - d[i] for i in range(3)]
    S = [1e-6 + x * x for x in d]
    D1 = e[0] * (4 / 3 * e[0] + d[1]) + S[1]
    D2 = e[1] * (4 / 3 * e[1] + d[1]) + S[1]
    D3 = e[2] * (4 / 3 * e[2] - d[2]) + S[2]
    c = weights(D1, D2, D3, abs(D1 - D3))
    return (V[2] + 0.5 * d[1]) + (c[0] * e[0] + c[1] * e[1] + c[2] * (3 * e[2 - 1] - e[2]))


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
