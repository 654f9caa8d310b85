"""The compaction's column sort at the edges of its tiles (1,024 columns), on
both sides of the number of tiles from which the digit counts are scanned by
a kernel (128), and for alphabets whose size packs a different number of
characters in a 64-bit key: whole numbers, so the result is exactly that of a
sort on the host."""
import numpy as np
import pytest

from crux_gb300 import Alignment, TaxaMap
from crux_gb300.compact import compact

pytestmark = pytest.mark.gpu

ALL = b"ACGTRYKMSWBDHVN-"


def host(rows, canon, freqs):
    cols = np.ascontiguousarray(canon[rows].T)
    order = np.lexsort(cols.T[::-1])
    cols, freqs = cols[order], freqs[order]
    first = np.ones(len(cols), dtype=bool)
    first[1:] = (cols[1:] != cols[:-1]).any(axis=1)
    return cols[first].T, np.add.reduceat(freqs, np.flatnonzero(first))


@pytest.mark.parametrize("ntaxa,nsites,alphabet,pool", [
    (7, 1023, b"ACGT", 300), (7, 1024, b"A", 1), (64, 1025, b"AC", 700),
    (27, 2048, b"ACGT-", 1500), (28, 2049, b"ACGT-", 1500), (130, 5000, ALL, 4000),
    (3, 131072, b"ACGTN", 100), (9, 131073, b"ACGTN", 131073), (40, 140001, ALL, 90000)])
def test_sorted_columns_match_a_host_sort(gpu, ntaxa, nsites, alphabet, pool):
    rng = np.random.default_rng([ntaxa, nsites])
    codes = np.frombuffer(alphabet, dtype=np.uint8)
    # Columns of a pool, most of them near one column: digits crowd.
    base = np.repeat(codes[rng.integers(len(codes), size=(ntaxa, 1))], pool, axis=1)
    hit = rng.random((ntaxa, pool)) < 0.1
    base[hit] = codes[rng.integers(len(codes), size=int(hit.sum()))]
    rows = np.ascontiguousarray(base[:, rng.integers(pool, size=nsites)])
    aln = Alignment(taxaMap=TaxaMap(["T%d" % i for i in range(ntaxa)]), rows=rows)
    freqs = np.ascontiguousarray(aln.freqs, dtype=np.uint32)
    want, wfreq = host(rows, np.asarray(aln.charType.get().canon_table, dtype=np.uint8),
                       freqs)
    got, gfreq, _ = compact(aln)
    assert got.shape == want.shape
    assert (got == want).all()
    assert (gfreq == wfreq).all()
