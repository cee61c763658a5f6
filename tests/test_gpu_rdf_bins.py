"""The FP32-decided pair histogram against the oracle where its decision can go wrong:
distances exactly on bin edges and on the cut-off (a unit lattice), ions in several images and
at the same place, triclinic and non-cubic cells, ion counts around the tiles of 32, 256 and
512 (two ions per thread from 12288 on), bins far finer than FP32 resolves, and a coordinate
that is not finite (its pairs are never counted).  Counts are whole numbers: equality."""
import numpy as np
import pytest

from mdff20_b200 import rdf
from oracle import oracle

pytestmark = pytest.mark.gpu


def _counts(cell, pos, nionit, cut, resg, nbins):
    with rdf.RDF(nionit, cut, resg, nbins) as acc:
        acc.add(cell, pos)
        return acc.counts()[0]


@pytest.mark.parametrize("resg", [0.1, 0.25, 1.0])
def test_edges_of_bins(resg):
    g = np.stack(np.meshgrid(*[np.arange(12.0)] * 3, indexing="ij"), -1).reshape(-1, 3) - 6.0
    cell, cut = np.eye(3) * 12.0, 6.0
    nionit, nbins = [700, 1028], int(cut / resg) + 1
    np.testing.assert_array_equal(_counts(cell, g, nionit, cut, resg, nbins),
                                  oracle.gr_counts([(cell, g)], nionit, cut, resg, nbins))


@pytest.mark.parametrize("n,tri,resg", [(1, False, 0.1), (2, True, 0.1), (33, True, 0.05), (257, False, 0.02),
                                        (511, True, 0.02), (1025, False, 1e-5), (12289, False, 0.1),
                                        (12300, True, 0.05)])
def test_sizes_and_cells(n, tri, resg):
    rng = np.random.default_rng(n)
    cell = np.diag([21.0, 26.0, 33.0])
    if tri:
        cell[1, 0], cell[2, 0], cell[2, 1] = 4.0, -3.0, 6.0
    pos = (rng.random((n, 3)) * 5.0 - 2.0) @ cell   # several images
    if n > 2:
        pos[n // 2] = pos[0]                          # the same place
    nionit = [n // 3, n - n // 3 - n // 5, n // 5]
    cut = 9.7
    nbins = min(int(cut / resg) + 1, 40000)
    np.testing.assert_array_equal(_counts(cell, pos, nionit, cut, resg, nbins),
                                  oracle.gr_counts([(cell, pos)], nionit, cut, resg, nbins))


def test_not_finite():
    rng = np.random.default_rng(3)
    cell, n = np.eye(3) * 15.0, 300
    pos = rng.random((n, 3)) * 15.0
    bad = pos.copy()
    bad[250, 1] = np.nan
    got = _counts(cell, bad, [200, 100], 7.0, 0.1, 71)
    want = oracle.gr_counts([(cell, np.delete(pos, 250, 0))], [200, 99], 7.0, 0.1, 71)
    np.testing.assert_array_equal(got, want)
