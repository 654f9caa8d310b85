"""The walker's own choice of launch shape (no cxgTune before it): for every
number of components a thread or a group of threads may hold, at pattern
counts around the warps, tiles and waves the choice is made by, lnL and site
lnLs agree with the FP64 oracle within the parity bars of each form (1e-11
and 1e-6 relative), and tuned shapes give the same bits.  This file is
collected before any that tunes: a tuned shape stays for the process."""
import numpy as np
import pytest

from crux_gb300 import Alignment, Lik, TaxaMap, Tree, synth, tune
from crux_gb300.batch import Batch
from crux_gb300.plan import Plan

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-11, "fp32": 1e-6}

# taxa, sites (not compacted: as many patterns, padded by the Lik).
SIZES = [(9, 5), (17, 129), (70, 1000), (5, 20011), (4, 47003), (4, 84000), (4, 98304),
         (4, 200001)]
# Gamma categories, +I: 1, 2, 3, 4, 5, 6, 7 and 8 components.
MODELS = [(1, 0.0), (2, 0.0), (3, 0.0), (4, 0.0), (4, 0.2), (6, 0.0), (6, 0.2),
          (8, 0.0)]
SEEN = {}


def make(ntaxa, nsites, ncat, pinv, lib, precision):
    rng = np.random.default_rng([ntaxa, nsites, ncat])
    newick = synth.yule_newick(ntaxa, 0.1, rng)
    codes = np.frombuffer(b"ACGT-RN", dtype=np.uint8)
    rows = codes[rng.choice(7, p=[.24, .24, .24, .24, .02, .01, .01],
                            size=(ntaxa, nsites))]
    aln = Alignment(taxaMap=TaxaMap(["T%d" % i for i in range(ntaxa)]), rows=rows)
    tree = Tree(newick)
    tree.deroot()
    tree.canonize(aln.taxaMap)
    lik = Lik(tree, aln, ncat=ncat, invar=pinv > 0.0, lib=lib, precision=precision)
    synth.apply_params(lik, 0, synth.gtr_params(rng), 0.5, pinv)
    return lik


def sizes_of(model):
    # The largest walks with the benchmark's components and with one.
    return [s for s in SIZES if s[1] < 40000 or model in ((1, 0.0), (4, 0.0))]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("model", MODELS)
def test_chosen_shape_matches_oracle(gpu, port, model, precision):
    ncat, pinv = model
    for ntaxa, nsites in sizes_of(model):
        lik = make(ntaxa, nsites, ncat, pinv, gpu, precision)
        got, site = lik.lnL(), lik.siteLnLs()
        ref = make(ntaxa, nsites, ncat, pinv, port, "fp64")
        want, wsite = ref.lnL(), np.array(ref.siteLnLs())
        assert abs(got - want) <= TOL[precision] * abs(want), (ntaxa, nsites)
        tol = 1e-10 if precision == "fp64" else 1e-4
        assert np.max(np.abs(np.array(site) - wsite) / np.abs(wsite)) <= tol
        edge = lik.tree.edges[ntaxa // 2]
        edge.length *= 1.5
        path = lik.lnL()
        plan = Plan(lik, precision)
        SEEN[model, precision, ntaxa, nsites] = (got, site, path, plan.shape())
        plan.close()


@pytest.mark.parametrize("nsites", [129, 84000])
def test_batch_of_one_takes_a_batched_shape(gpu, port, nsites):
    """A batch of one job, at sizes where a plan takes the small tiles and
    where it takes the wide build, which batches do not have."""
    lik = make(5, nsites, 4, 0.0, gpu, "fp32")
    ref = make(5, nsites, 4, 0.0, port, "fp64")
    lik.prepare_plan()
    b = Batch([lik], "fp32")
    got, want = b.run()[0], ref.lnL()
    b.close()
    assert abs(got - want) <= TOL["fp32"] * abs(want)


def test_chosen_shapes_differ_and_tuned_ones_give_their_bits(gpu):
    """Runs after the choices above: the process is tuned from here on."""
    if not SEEN:
        pytest.skip("needs the chosen shapes' results")
    shapes = {(s["tile"], s["threads_per_pattern"]) for _, _, _, s in SEEN.values()}
    assert len(shapes) >= 4, shapes
    for (model, precision, ntaxa, nsites), (got, site, path, _) in SEEN.items():
        if nsites > 40000:
            continue
        for shape in ((64, 1, 1, 24 << 10), (32, 1, 1, 0), (128, 1, 1, 48 << 10)):
            tune.set_shape(gpu, *shape)
            lik = make(ntaxa, nsites, *model, gpu, precision)
            assert lik.lnL() == got, (model, precision, ntaxa, nsites, shape)
            assert lik.siteLnLs() == site
            edge = lik.tree.edges[ntaxa // 2]
            edge.length *= 1.5
            assert lik.lnL() == path
