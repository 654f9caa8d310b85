"""Gamma categories computed on the device: shapes on both sides of every
branch of the quantile (start values, series or continued fraction, a
series longer than the 16 terms taken at once), for category counts that
leave warps idle and that take more than one turn.  The server builds the
model on the device, the oracle's rates come from the host's routines.

Tolerance: both stop the incomplete Gamma ratio at 1e-10, so a cut is off by
some 1e-10 and a rate, a difference of two cuts times the number of
categories, by 2e-9 at most; the lnL moves relatively by no more than a few
times that: 1e-8."""
import numpy as np
import pytest

from crux_gb300 import synth
from crux_gb300.serve import LNL, PreparedRequest, Server

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncat", [2, 3, 4, 5, 8])
def test_rates_match_the_hosts(gpu, port, ncat):
    case = synth.Case(9, 150, 0.1, 77)
    case.ncat = ncat
    srv = Server("fp64")
    got, want = [], []
    for alpha in (0.02, 0.07, 0.15, 0.161, 0.3, 0.5, 0.999, 1.0, 1.7, 5.0, 40.0, 300.0):
        case.alpha = alpha
        got.append(srv.wait(srv.submit(PreparedRequest(case, LNL)))[0])
        want.append(case.lik(port).lnL())
    srv.close()
    got, want = np.array(got), np.array(want)
    assert np.max(np.abs(got - want) / np.abs(want)) <= 1e-8, got - want
