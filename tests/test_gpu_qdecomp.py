"""The device eigensystem at the models where Jacobi rotations can go wrong:
equal rates and frequencies (every eigenvalue but one the same), rates over
many orders of magnitude, a zero rate, one dominating frequency.  P(t) from
the cube and eigenvalues against a Taylor series of expm in extended
precision.

Tolerance: an entry of P is a sum of four products of cube entries (three
roundings each) and exponentials (one each), with |cube| <= sqrt(pi_max /
pi_min) and the rotations orthogonal to a few eps, so about 40 eps times that
factor: 40 * 2.2e-16 * sqrt(pi_max / pi_min)."""
import ctypes

import numpy as np
import pytest

from crux_gb300 import _abi

pytestmark = pytest.mark.gpu


def expm(Q, t):
    A = Q.astype(np.longdouble) * np.longdouble(t)
    s = max(0, int(np.ceil(np.log2(max(1e-9, float(np.abs(A).sum(1).max())))))) + 6
    A = A / np.longdouble(2) ** s
    P = np.eye(4, dtype=np.longdouble)
    term = np.eye(4, dtype=np.longdouble)
    for k in range(1, 25):
        term = term @ A / k
        P = P + term
    for _ in range(s):
        P = P @ P
    return P


def models():
    rng = np.random.default_rng(41)
    yield np.ones(6), np.full(4, 0.25)
    yield np.ones(6), np.array([0.4, 0.3, 0.2, 0.1])
    yield np.array([1.0, 2.0, 1.0, 1.0, 2.0, 1.0]), np.full(4, 0.25)
    yield np.array([1.0, 0.0, 1.0, 1.0, 0.5, 1.0]), np.array([0.3, 0.3, 0.2, 0.2])
    yield np.ones(6), np.array([0.97, 0.01, 0.01, 0.01])
    for spread in (1e1, 1e2, 1e3, 1e4):
        for _ in range(8):
            yield (np.exp(rng.uniform(-0.5, 0.5, 6) * np.log(spread)),
                   rng.dirichlet(np.full(4, 2.0)))


def test_eigensystem_gives_expm(gpu):
    for rates, freqs in models():
        r, f = np.ascontiguousarray(rates), np.ascontiguousarray(freqs)
        pn, cube, ev = np.zeros(4), np.zeros(64), np.zeros(4)
        qn = ctypes.c_double()
        assert not gpu.CxLikQDecomp(4, _abi.dptr(r), _abi.dptr(f), _abi.dptr(pn),
                                    ctypes.byref(qn), _abi.dptr(cube), _abi.dptr(ev))
        assert np.allclose(pn, f / f.sum(), rtol=4e-16, atol=0)
        R = np.zeros((4, 4))
        R[np.triu_indices(4, 1)] = r
        R = R + R.T
        Q = R * pn[None, :]
        np.fill_diagonal(Q, 0.0)
        np.fill_diagonal(Q, -Q.sum(1))
        mean = -(pn * np.diag(Q)).sum()
        assert abs(qn.value * mean - 1.0) <= 1e-14
        tol = 40 * 2.2e-16 * np.sqrt(pn.max() / pn.min())
        for t in (0.0, 1e-3, 0.1, 1.0, 10.0):
            v = t * qn.value
            P = np.einsum("ijk,k->ij", cube.reshape(4, 4, 4), np.exp(ev * v))
            assert np.abs(P - expm(Q, v)).max() <= tol, (rates, freqs, t)
