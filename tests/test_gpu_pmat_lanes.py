"""P matrices by sixteen lanes (plans of few child edges) and by four: both
sides of the limit give the bits of the batched kernel, which uses four."""
import numpy as np
import pytest

from crux_gb300 import Alignment, Lik, TaxaMap, Tree, synth
from crux_gb300.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("ntaxa,ncat,pinv", [
    (5, 1, 0.0), (9, 3, 0.0), (9, 6, 0.2), (129, 4, 0.0), (130, 4, 0.0), (257, 1, 0.0),
    (258, 1, 0.0), (240, 4, 0.2)])
def test_plan_equals_batch_bits(gpu, ntaxa, ncat, pinv, precision):
    rng = np.random.default_rng([ntaxa, ncat])
    codes = np.frombuffer(b"ACGT-RYN", dtype=np.uint8)
    rows = codes[rng.integers(8, size=(ntaxa, 130))]
    aln = Alignment(taxaMap=TaxaMap(["T%d" % i for i in range(ntaxa)]), rows=rows)
    tree = Tree(synth.yule_newick(ntaxa, 0.1, rng))
    tree.deroot()
    tree.canonize(aln.taxaMap)
    lik = Lik(tree, aln, ncat=ncat, invar=pinv > 0.0, lib=gpu, precision=precision)
    synth.apply_params(lik, 0, synth.gtr_params(rng), 0.5, pinv)
    got = lik.lnL()
    lik.prepare_plan()
    b = Batch([lik], precision)
    want = b.run()[0]
    b.close()
    assert got == want
