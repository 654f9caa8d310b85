"""Every path that takes the library's own launch shapes, with no shape set: nodes
of many children, internal roots, mixtures, batches of many jobs, chains alone
and several together, and a server's requests of different shapes in one burst,
at sizes on both sides of the sizes the choice is made by.  Within the parity
bars of each form against the FP64 oracle (1e-11 and 1e-6 relative)."""
import numpy as np
import pytest

from crux_gb300 import Alignment, Lik, TaxaMap, Tree, synth, tune
from crux_gb300.batch import Batch
from crux_gb300.mc3 import Mc3
from crux_gb300.serve import LNL, PreparedRequest, Server

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-11, "fp32": 1e-6}
POLY = ("(T0:.1,T1:.2,(T2:.1,T3:.3,T4:.05,T5:.2,(T6:.1,(T7:.2,T8:.3):.1):.1):.15,"
        "(T9:.05,(T10:.4,T11:.1,T12:.2,T13:.1,T14:.3,T15:.2):.1):.2);")


@pytest.fixture(autouse=True)
def automatic(gpu):
    assert tune.get(gpu) == tune.AUTO
    yield
    assert tune.get(gpu) == tune.AUTO


def close(got, want, precision):
    assert abs(got - want) <= TOL[precision] * abs(want), (got, want)


def make(newick, nsites, lib, precision, ncat=4, pinv=0.0, nmodels=1):
    """Random columns, as many patterns as sites."""
    rng = np.random.default_rng([nsites, ncat, nmodels])
    n = newick.count("T")
    rows = np.frombuffer(b"ACGT-RN", dtype=np.uint8)[
        rng.choice(7, p=[.24, .24, .24, .24, .02, .01, .01], size=(n, nsites))]
    aln = Alignment(taxaMap=TaxaMap(["T%d" % i for i in range(n)]), rows=rows)
    tree = Tree(newick)
    tree.deroot()
    tree.canonize(aln.taxaMap)
    lik = Lik(tree, aln, nmodels=nmodels, ncat=ncat, invar=pinv > 0.0, lib=lib,
              precision=precision)
    for i in range(nmodels):
        synth.apply_params(lik, i, synth.gtr_params(rng), 0.5 if ncat > 1 else None, pinv)
        lik.setWeight(i, 1.0 + i)
    return lik


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("nsites", [40, 3000, 25000, 45000, 84000])
def test_polytomies_and_inner_roots(gpu, port, precision, nsites):
    ref, lik = make(POLY, nsites, port, "fp64"), make(POLY, nsites, gpu, precision)
    close(lik.lnL(), ref.lnL(), precision)
    for at in (3, 11, 17):
        close(lik.lnL(lik.tree.nodes[at]), ref.lnL(ref.tree.nodes[at]), precision)
    for k in (ref, lik):
        k.tree.edges[6].length *= 2.0
    close(lik.lnL(), ref.lnL(), precision)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("ncat, nmodels", [(4, 2), (3, 2), (2, 4), (1, 3), (1, 7)])
@pytest.mark.parametrize("nsites", [300, 25000])
def test_mixtures(gpu, port, precision, ncat, nmodels, nsites):
    out = []
    for lib, prec in ((port, "fp64"), (gpu, precision)):
        k = make(POLY, nsites, lib, prec, ncat, nmodels=nmodels)
        v = [k.lnL()]
        k.tree.edges[4].length *= 1.5
        out.append(v + [k.lnL()])
    for got, want in zip(out[1], out[0]):
        close(got, want, precision)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("ncat, pinv", [(1, 0.0), (4, 0.0), (4, 0.2)])
@pytest.mark.parametrize("njobs, top", [(2, 400), (9, 3000), (24, 9000)])
def test_batches_of_many_jobs(gpu, port, precision, ncat, pinv, njobs, top):
    sizes = [int(60 * (top / 60) ** (j / (njobs - 1))) for j in range(njobs)]
    rng = np.random.default_rng(njobs)
    trees = [synth.yule_newick(int(rng.integers(5, 60)), 0.1, rng) for _ in sizes] \
        if njobs != 9 else [POLY] * 9
    want = [make(t, n, port, "fp64", ncat, pinv).lnL() for t, n in zip(trees, sizes)]
    liks = [make(t, n, gpu, precision, ncat, pinv) for t, n in zip(trees, sizes)]
    for k in liks:
        k.prepare_plan()
    b = Batch(liks, precision)
    got = b.run()
    b.close()
    for g, w in zip(got, want):
        close(g, w, precision)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("ncat, pinv", [(1, 0.0), (2, 0.0), (4, 0.0), (4, 0.2)])
@pytest.mark.parametrize("nchains, nsites", [(1, 200), (1, 30000), (5, 1000), (3, 30000)])
def test_chains(gpu, port, precision, ncat, pinv, nchains, nsites):
    """The lnL a run starts from and, from its states after some moves, the lnL
    that the oracle gives the chains' trees and models."""
    case = synth.Case(14, nsites, 0.2, 21, alpha=0.5 if ncat > 1 else None, ncat=ncat, pinv=pinv)
    aln = case.alignment()
    m = Mc3(case.tree(aln.taxaMap), aln, case.params["rates"], case.params["freqs"],
            alpha=case.alpha, ncat=ncat, pinv=pinv, nchains=nchains, seed=4,
            moves={"brlen": 1.0, "nni": 1.0, "spr": 1.0, "rates": 0.5,
                   "alpha": 0.5 if ncat > 1 else 0.0},
            precision=precision, graph_gens=4)
    try:
        want = case.lik(lib=port, alignment=aln).lnL()
        for i in range(nchains):
            close(m.chain_state(i)["lnL"], want, precision)
        m.run(24)
        from crux_gb300.mc3 import newick_from_arrays
        for i in range(nchains):
            st = m.chain_state(i)
            tree = Tree(newick_from_arrays(st["parent"], st["len"], aln.taxaMap.taxa))
            tree.deroot()
            tree.canonize(aln.taxaMap)
            ref = Lik(tree, aln, ncat=ncat, invar=pinv > 0.0, lib=port, precision="fp64")
            synth.apply_params(ref, 0, {"rates": st["rates"], "freqs": st["freqs"]},
                               st["alpha"] if ncat > 1 else None, pinv)
            # (The Gamma quantiles of chain and Lik agree to the 5e-7 of
            # their iteration.)
            tol = TOL[precision] if st["alpha"] == case.alpha or ncat == 1 else \
                max(TOL[precision], 1e-6)
            assert abs(st["lnL"] - ref.lnL()) <= tol * abs(ref.lnL())
    finally:
        m.close()


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_a_burst_of_shapes(gpu, port, precision):
    """Requests of one, two and four threads a pattern in the FP64 form, and of
    different components, served together."""
    cases = [synth.Case(9, 300, 0.2, 1), synth.Case(18, 40000, 0.4, 2),
             synth.Case(12, 900, 0.2, 3, alpha=None), synth.Case(12, 900, 0.2, 4, ncat=2),
             synth.Case(12, 700, 0.2, 5, pinv=0.2), synth.Case(14, 30000, 0.4, 6, ncat=3)]
    reqs = [PreparedRequest(c, LNL) for c in cases]
    assert {r.req.npat > 19456 for r in reqs} == {True, False}
    srv = Server(precision)
    try:
        tickets = [srv.submit(r) for r in reqs * 3]
        got = [srv.wait(t)[0] for t in tickets]
    finally:
        srv.close()
    for i, r in enumerate(reqs):
        close(got[i], r.oracle_lik(port).lnL(), precision)
        assert got[i + len(reqs)] == got[i] and got[i + 2 * len(reqs)] == got[i]
