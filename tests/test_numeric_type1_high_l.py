"""Numeric type 1 integrals of shells up to L = 10 (L_A + L_B <= 12) against the three-centre Gaussian
integral <A| exp(-zeta r_C^2) |B>, a product of one-dimensional integrals that Gauss-Hermite
quadrature gives exactly: a U_L of r^0 terms directly, the Gaussian nucleus as
-Z 2/sqrt(pi) int_0^sqrt(xi) exp(-u^2 r^2) du.

Tolerance: the path sums radial integrals of positive terms, at most 8191 of them, each sum good to
8191 eps = 1e-12 of itself, times the angular factors (their moduli add up to at most
sum_lambda (2 lambda + 1) <= 91 for lambda of one parity up to 12) and the binomial factors. The sum
of the moduli of the binomial terms is bounded with the largest radial factor, lambda = 0."""
import math

import numpy as np
import pytest

from libgrpp_b200.system import GRPP, Potential, Shell, System

GAUSS = 2  # LIBGRPP_NUCLEAR_MODEL_GAUSSIAN
CLASSES = [(8, 4), (4, 8), (8, 0), (9, 3), (10, 2), (2, 10), (0, 10), (7, 5), (6, 6)]


def _powers(L):
    return [(L - k, k - v, v) for k in range(L + 1) for v in range(k + 1)]  # libgrpp's order


def _norm(L, a):  # norm_gaussian.c:16-23, no double-factorial term
    return (2 * a / math.pi) ** 0.75 * (4 * a) ** (L / 2)


def _axis(a, b, z, A, B, C, la, lb):
    x, w = np.polynomial.hermite.hermgauss((la + lb) // 2 + 1)
    q = a + b + z
    Q = (a * A + b * B + z * C) / q
    K = math.exp(-(a * b * (A - B) ** 2 + a * z * (A - C) ** 2 + b * z * (B - C) ** 2) / q) / math.sqrt(q)
    x = Q + x / math.sqrt(q)
    return K * np.einsum("ik,jk,k->ij", [(x - A) ** i for i in range(la + 1)], [(x - B) ** j for j in range(lb + 1)], w)


def _block(A, B, C, zetas, weights):
    """sum_k weights_k <A| exp(-zetas_k r_C^2) |B> over contracted normalised shells."""
    out = np.zeros((len(_powers(A.L)), len(_powers(B.L))))
    for ca, a in zip(A.coeffs, A.alpha):
        for cb, b in zip(B.coeffs, B.alpha):
            f = ca * cb * _norm(A.L, a) * _norm(B.L, b)
            for z, w in zip(zetas, weights):
                t = [_axis(a, b, z, A.origin[d], B.origin[d], C[d], A.L, B.L) for d in range(3)]
                out += f * w * np.array([[t[0][i[0], j[0]] * t[1][i[1], j[1]] * t[2][i[2], j[2]] for j in _powers(B.L)]
                                         for i in _powers(A.L)])
    return out


def _moduli(A, B, C, zetas, weights):
    """Bound of the summed moduli of every element: int |V| exp(k r - ..) (r + |CA_x|)^i .. dr, lambda = 0."""
    r = np.linspace(0.0, 12.0, 4001)
    h = r[1] - r[0]
    V = np.abs(sum(w * np.exp(-z * r * r) for z, w in zip(zetas, weights)))
    CA, CB = np.abs(C - A.origin), np.abs(C - B.origin)
    out = np.zeros((len(_powers(A.L)), len(_powers(B.L))))
    for ca, a in zip(A.coeffs, A.alpha):
        for cb, b in zip(B.coeffs, B.alpha):
            k = 2 * np.linalg.norm(a * (C - A.origin) + b * (C - B.origin))
            g = abs(ca * cb) * _norm(A.L, a) * _norm(B.L, b) * V * r * r * np.exp(k * r - (a + b) * r * r - a * CA @ CA - b * CB @ CB)
            for m, i in enumerate(_powers(A.L)):
                for n, j in enumerate(_powers(B.L)):
                    p = np.prod([(r + CA[d]) ** i[d] * (r + CB[d]) ** j[d] for d in range(3)], axis=0)
                    out[m, n] += 4 * math.pi * h * np.sum(g * p)
    return out


def _system(la, lb):
    rng = np.random.default_rng(100 * la + lb)
    A = Shell(np.array([0.35, -0.25, 0.3]), la, [0.7, 0.4], [0.5, 1.1])
    B = Shell(np.array([-0.2, 0.45, 0.15]), lb, [0.9], [0.8])
    U = Potential(0, 0, [2, 2], [1.5, -0.6], [0.9, 2.0])
    C = [(np.array([0.05, 0.1, -0.15]), 0), (rng.uniform(-0.4, 0.4, 3), 0)]
    return System(shells=[A, B], grpps=[GRPP(UL=U)], centres=C), A, B, U


def _check(got, S, A, B, potentials):
    got = got.reshape(len(S.centres), len(_powers(A.L)), len(_powers(B.L)))
    for blk, (C, _), (z, w) in zip(got, S.centres, potentials):
        want = _block(A, B, C, z, w)
        tol = 91 * 1e-12 * _moduli(A, B, C, z, w)
        assert np.abs(want).max() > 1e3 * np.median(tol), "the comparison would be empty"
        assert np.all(np.abs(blk - want) <= tol), float((np.abs(blk - want) / tol).max())


def _batch(S):
    n = len(S.centres)
    return S.batch(np.zeros(n, np.int32), np.ones(n, np.int32), np.arange(n, dtype=np.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("la,lb", CLASSES)
def test_local_potential(gpu_lib, la, lb):
    S, A, B, U = _system(la, lb)
    got = gpu_lib.type1_numeric_batch(_batch(S))
    _check(got, S, A, B, [(np.array(U.alpha), np.array(U.coeffs))] * len(S.centres))


@pytest.mark.gpu
@pytest.mark.parametrize("la,lb", CLASSES)
def test_gaussian_nucleus(gpu_lib, la, lb):
    S, A, B, _ = _system(la, lb)
    Z, rms = np.array([3.0, 8.0]), np.array([0.4, 0.6])
    got = gpu_lib.nuclear_attraction_batch(_batch(S), GAUSS, Z, np.stack([rms, 0 * rms, 0 * rms], 1))
    x, w = np.polynomial.legendre.leggauss(48)
    pots = []
    for q, R in zip(Z, rms):
        top = math.sqrt(1.5) / R
        u = 0.5 * top * (x + 1)
        pots.append((u * u, -q * 2 / math.sqrt(math.pi) * 0.5 * top * w))
    _check(got, S, A, B, pots)
