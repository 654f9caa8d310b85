"""2^28 patterns, from where a row of a CL no longer lies within 32 bits of
bytes of the next: a chain on a block of patterns repeated has the lnL of the
block times the repeats.  (Two components: two units a row; the root reads its
internal child back from memory.  35 GB on the device.)"""
import types

import numpy as np
import pytest

from crux_gb300 import TaxaMap, Tree
from crux_gb300.mc3 import Mc3

pytestmark = pytest.mark.gpu


def chain_lnl(masks):
    """The lnL a chain starts from, on leaf state masks [taxa][patterns]."""
    names = TaxaMap(["T%d" % i for i in range(len(masks))])
    same = types.SimpleNamespace(val_table=np.arange(16, dtype=np.uint8))
    aln = types.SimpleNamespace(taxaMap=names, rows=masks, nchars=masks.shape[1],
                                charType=types.SimpleNamespace(get=lambda: same),
                                freqs=np.ones(masks.shape[1], dtype=np.uint32))
    tree = Tree("(T0:0.1,T1:0.3,(T2:0.2,T3:0.1):0.2);")
    tree.deroot()
    tree.canonize(names)
    m = Mc3(tree, aln, [1.0, 2.0, 1.0, 1.5, 2.0, 1.0], [0.3, 0.2, 0.3, 0.2], alpha=0.5, ncat=2,
            nchains=1, precision="fp32", graph_gens=1)
    try:
        return m.chain_state(0)["lnL"]
    finally:
        m.close()


def test_rows_past_32_bits(gpu):
    rng = np.random.default_rng(3)
    block = (1 << rng.integers(4, size=(4, 1 << 14))).astype(np.uint8)
    repeats = 1 << 14
    want = chain_lnl(block)
    assert np.isfinite(want)
    got = chain_lnl(np.tile(block, (1, repeats)))
    assert abs(got - want * repeats) <= 1e-12 * abs(want * repeats)
