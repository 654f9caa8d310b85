"""The units of the exchangeabilities do not matter to the eigensystem: rates
times 2^k give the same eigenvectors, the eigenvalues times 2^k and the
normaliser times 2^-k, bit for bit, over the range in which these are normal
numbers."""
import ctypes

import numpy as np
import pytest

from crux_gb300 import _abi

pytestmark = pytest.mark.gpu


def decompose(gpu, rates, freqs):
    pn, cube, ev = np.zeros(4), np.zeros(64), np.zeros(4)
    qn = ctypes.c_double()
    rc = gpu.CxLikQDecomp(4, _abi.dptr(np.ascontiguousarray(rates)),
                          _abi.dptr(np.ascontiguousarray(freqs)), _abi.dptr(pn),
                          ctypes.byref(qn), _abi.dptr(cube), _abi.dptr(ev))
    return rc, pn, qn.value, cube, ev


@pytest.mark.parametrize("k", [-1000, -700, -530, -515, -400, -52, 40, 400, 505, 515, 700, 1000])
@pytest.mark.parametrize("model", [0, 1])
def test_rates_in_any_unit(gpu, model, k):
    rng = np.random.default_rng(model)
    rates = np.exp(rng.uniform(-2, 2, 6)) if model else np.array([1., 2., 1., 1., 2., 1.])
    freqs = rng.dirichlet(np.full(4, 3.0))
    rc, pn, qn, cube, ev = decompose(gpu, rates, freqs)
    assert not rc
    rc, pn2, qn2, cube2, ev2 = decompose(gpu, np.ldexp(rates, k), freqs)
    assert not rc
    assert np.array_equal(pn, pn2) and np.array_equal(cube, cube2)
    assert qn2 == np.ldexp(qn, -k)
    # (The zero eigenvalue is a rounding error, subnormal at the low end.)
    tiny = np.abs(np.ldexp(ev, k)) < 2.0 ** -1020
    assert np.array_equal(ev2[~tiny], np.ldexp(ev, k)[~tiny])
    assert np.all(np.abs(ev2[tiny]) < 2.0 ** -1019)
