"""Counts of both orders of a pair from a histogram that holds each pair once: one to four types, bins
that just fit the block's shared counters (10240) and that do not, two configurations added up.  Bins
so fine that every pair is decided in FP64 (triclinic cells: 0.004 A), at ion counts around the tiles
of 256.  Whole numbers: equality with the oracle."""
import numpy as np
import pytest

from mdff20_b200.rdf import RDF
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nionit", [[700], [300, 401], [100, 1, 600], [200, 200, 0, 301]])
@pytest.mark.parametrize("past", [0, 1])
def test_both_orders(nionit, past):
    rng = np.random.default_rng(len(nionit))
    n, cell, cut = sum(nionit), np.eye(3) * 17.0, 8.0
    nbins = 10240 // len(nionit) ** 2 + past
    frames = [(cell, rng.random((n, 3)) * 17.0) for _ in range(2)]
    resg = cut / nbins * 1.0001
    with RDF(nionit, cut, resg=resg, nbins=nbins) as acc:
        for c, p in frames:
            acc.add(c, p)
        got, nconf = acc.counts()[:2]
        again = acc.counts()[0]
    assert nconf == 2
    np.testing.assert_array_equal(got, oracle.gr_counts(frames, nionit, cut, resg, nbins))
    np.testing.assert_array_equal(got, again)


@pytest.mark.parametrize("n", [1, 2, 31, 255, 256, 257, 513, 1300])
@pytest.mark.parametrize("nbins", [2000, 2500, 2600])   # either side of the chance of an open pair, of 10240 counters
def test_fine_bins(n, nbins):
    rng = np.random.default_rng(n)
    cell = np.array([[21.0, 0.0, 0.0], [4.0, 26.0, 0.0], [-3.0, 6.0, 33.0]])
    pos = (rng.random((n, 3)) * 5.0 - 2.0) @ cell
    nionit = [n // 3, n - n // 3]
    cut = 9.7
    resg = cut / nbins * 1.0001
    with RDF(nionit, cut, resg=resg, nbins=nbins) as acc:
        acc.add(cell, pos)
        got = acc.counts()[0]
    np.testing.assert_array_equal(got, oracle.gr_counts([(cell, pos)], nionit, cut, resg, nbins))


@pytest.mark.parametrize("n", [8897, 9025])   # tiles of 64, more of them than blocks per SM
@pytest.mark.parametrize("nbins", [2500, 2600])   # either side of 10240 counters
def test_fine_bins_many_tiles(n, nbins):
    rng = np.random.default_rng(n)
    cell = np.array([[51.0, 0.0, 0.0], [4.0, 56.0, 0.0], [-3.0, 6.0, 53.0]])
    pos = (rng.random((n, 3)) * 5.0 - 2.0) @ cell
    nionit = [n // 3, n - n // 3]
    cut = 9.7
    resg = cut / nbins * 1.0001
    with RDF(nionit, cut, resg=resg, nbins=nbins) as acc:
        acc.add(cell, pos)
        got = acc.counts()[0]
    np.testing.assert_array_equal(got, oracle.gr_counts([(cell, pos)], nionit, cut, resg, nbins))
