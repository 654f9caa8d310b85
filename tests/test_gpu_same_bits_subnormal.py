"""Every shape gives the same bits also where rows hold subnormal entries: the
FP32 form rescales patterns in groups, which must not depend on how many of
them a warp, a thread or a tile holds.  Pairs of equal or different leaves
spread the rows of two rate categories over 2^90 to 2^150, patterns that need
a rescale early lie among ones that do not, and a clade that favours the other
category brings the small entries back."""
import numpy as np
import pytest

from crux_gb300 import Alignment, Lik, TaxaMap, Tree, tune

pytestmark = pytest.mark.gpu

PAIRS, STEADY, MIXED = 16, 60, 6


def chain(parts, t):
    text = parts[0]
    for p in parts[1:]:
        text = "(%s,%s):%r" % (text, p, t)
    return text


def make(gpu, ncat, nsites=1000):
    rng = np.random.default_rng(ncat)
    n = 1 + 2 * PAIRS + STEADY + MIXED
    rows = np.full((n, nsites), ord("A"), dtype=np.uint8)
    nmis = rng.integers(6, PAIRS + 1, size=nsites)
    for k in range(PAIRS):
        rows[2 + 2 * k, nmis > k] = ord("C")
    # A few leaves at random, in one pattern of five.
    some = np.flatnonzero(rng.random(nsites) < 0.2)
    for k in range(n - MIXED, n):
        rows[k, some] = rng.choice(np.frombuffer(b"ACGT", dtype=np.uint8), size=len(some))
    aln = Alignment(taxaMap=TaxaMap(["T%d" % i for i in range(n)]), rows=rows)
    leaf = iter(range(1, n))
    pairs = ["(T%d:0.5,T%d:0.5):0.01" % (next(leaf), next(leaf)) for _ in range(PAIRS)]
    steady = ["T%d:5.0" % next(leaf) for _ in range(STEADY)]
    mixed = ["T%d:0.001" % next(leaf) for _ in range(MIXED)]
    tree = Tree("((%s,%s):0.01,%s,T0:0.1);" % (chain(mixed, 0.001), chain(pairs, 0.01),
                                               chain(steady, 0.01)))
    tree.deroot()
    tree.canonize(aln.taxaMap)
    lik = Lik(tree, aln, ncat=ncat, lib=gpu, precision="fp32")
    lik.setAlpha(0, 0.11)
    return lik


@pytest.mark.parametrize("ncat", [2, 4])
def test_every_shape_same_bits(gpu, ncat):
    saved = tune.get(gpu)
    try:
        first = None
        for shape in tune.choices("fp32", ncat, budgets=(0, 24 << 10)):
            tune.set_shape(gpu, *shape)
            got = make(gpu, ncat).siteLnLs()
            first = first or got
            assert got == first, (shape, [i for i, (a, b) in enumerate(zip(got, first))
                                          if a != b][:8])
    finally:
        tune.set_shape(gpu, *saved)
