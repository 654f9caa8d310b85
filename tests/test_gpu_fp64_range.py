"""Range of the FP64 form: two clades that favour different mixture components
by more than 2^-700 each, joined at one branch.  The reference's scaling keeps
both components (its rows stay near 1); a row left near 2^-256 before the join
would lose them below the subnormals and make the site -inf.  Sites with 0 to
all of the mismatches, in tuned shapes and the library's own: lnL and site
lnLs within the parity bars of the form (1e-11 and 1e-10 relative)."""
import numpy as np
import pytest

from crux_gb300 import Alignment, Lik, TaxaMap, Tree, tune

pytestmark = pytest.mark.gpu

# Leaves: mismatched or equal pairs (a mismatch costs the slow category 2^12
# and the fast one 2^2), steady ones (each costs the fast one 2^2) and, in their
# clade, flat ones (each costs both 2^2; no longer than it takes, since a long
# branch multiplies the rounding of the zero eigenvalue).
PAIRS, STEADY, FLAT = 70, 400, 110


def balanced(parts, t):
    while len(parts) > 1:
        nxt = ["(%s,%s):%r" % (a, b, t) for a, b in zip(parts[::2], parts[1::2])]
        parts = nxt + parts[len(nxt) * 2:]
    return parts[0]


def make(lib):
    n = 1 + 2 * PAIRS + STEADY + FLAT
    # Site s has s mismatched pairs; everything else is constant.
    rows = np.full((n, PAIRS + 1), ord("A"), dtype=np.uint8)
    for s in range(PAIRS + 1):
        rows[2:1 + 2 * s:2, s] = ord("C")
    aln = Alignment(taxaMap=TaxaMap(["T%d" % i for i in range(n)]), rows=rows)
    leaf = iter(range(1, n))
    pairs = ["(T%d:0.5,T%d:0.5):0.01" % (next(leaf), next(leaf)) for _ in range(PAIRS)]
    steady = ["T%d:5.0" % next(leaf) for _ in range(STEADY)]
    flat = ["T%d:4e4" % next(leaf) for _ in range(FLAT)]
    newick = "(%s,%s,T0:0.1);" % (balanced(pairs, 0.01), balanced(steady + flat, 0.01))
    tree = Tree(newick)
    tree.deroot()
    tree.canonize(aln.taxaMap)
    lik = Lik(tree, aln, ncat=2, lib=lib, precision="fp64")
    lik.setAlpha(0, 0.11)
    return lik


def test_conflicting_components_keep_their_rows(gpu, port):
    ref = make(port)
    want, wsite = ref.lnL(), np.array(ref.siteLnLs())
    assert np.all(np.isfinite(wsite))
    saved = tune.get(gpu)
    try:
        for shape in (saved, (32, 1, 1, 0, 1), (64, 1, 1, 48 << 10, 1)):
            tune.set_shape(gpu, *shape)
            lik = make(gpu)
            site = np.array(lik.siteLnLs())
            assert np.max(np.abs(site - wsite) / np.abs(wsite)) <= 1e-10, shape
            lik.lik.invalidate = True
            assert abs(lik.lnL() - want) <= 1e-11 * abs(want)
    finally:
        tune.set_shape(gpu, *saved)
