"""Op lanes on nodes of many children: every degree a node may have gives the
bits of one lane, and the FP64 oracle's lnL and site lnLs within the FP32
parity bar (1e-6 relative; sites 1e-4).  Each child of the wide node is a clade
of leaves in conflict, whose rows have just been rescaled to 2^19 or more, so
that an unscaled product of seven of them would leave the FP32 range."""
import math

import numpy as np
import pytest

from crux_gb300 import Alignment, Lik, TaxaMap, Tree, synth, tune
from crux_gb300.plan import Plan

pytestmark = pytest.mark.gpu

CLADE = 5


@pytest.fixture
def restore(gpu):
    saved = tune.get(gpu)
    yield
    tune.set_shape(gpu, *saved)


def make(nkids, pinv, lib, precision):
    rng = np.random.default_rng([nkids, 41])
    codes = np.frombuffer(b"ACGT-", dtype=np.uint8)
    n = CLADE * nkids
    rows = codes[rng.choice(5, p=[.24, .24, .24, .24, .04], size=(n, 500))]
    aln = Alignment(taxaMap=TaxaMap(["T%d" % i for i in range(n)]), rows=rows)

    def clade(k):
        text = "T%d:0.05" % (CLADE * k)
        for j in range(1, CLADE):
            text = "(%s,T%d:0.05):0.05" % (text, CLADE * k + j)
        return text

    tree = Tree("(%s);" % ",".join(clade(k) for k in range(nkids)))
    tree.deroot()
    tree.canonize(aln.taxaMap)
    lik = Lik(tree, aln, ncat=4, invar=pinv > 0.0, lib=lib, precision=precision)
    synth.apply_params(lik, 0, synth.gtr_params(rng), 0.5, pinv)
    return lik


@pytest.mark.parametrize("pinv", [0.0, 0.2])
@pytest.mark.parametrize("nkids", list(range(4, 18)))
def test_wide_nodes_same_bits(gpu, port, restore, nkids, pinv):
    ref = make(nkids, pinv, port, "fp64")
    want, wsite = ref.lnL(), np.array(ref.siteLnLs())
    # The plan is rooted inside one clade: the others are the node's children.
    ref.lik.invalidate = True
    ref._prep(None)
    assert max(ntrail for _, ntrail, _ in ref.steps()) + 1 == nkids - 1
    out = []
    for lanes in (1, 2):
        tune.set_shape(gpu, 64, 1, 1, 24 << 10, lanes)
        lik = make(nkids, pinv, gpu, "fp32")
        lik._prep(None)
        plan = Plan(lik, "fp32")
        assert plan.shape()["lanes"] == lanes
        plan.close()
        lik.lik.invalidate = True
        out.append((lik.lnL(), lik.siteLnLs()))
    one, two = out
    for v, s in (one, two):
        assert math.isfinite(v)
        assert abs(v - want) <= 1e-6 * abs(want), (v, want)
        assert np.max(np.abs(np.array(s) - wsite) / np.abs(wsite)) <= 1e-4
    assert two == one
