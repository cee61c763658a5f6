"""Counts of both orders of a pair from a histogram that holds each pair once: one to four types, bins
that just fit the block's shared counters (10240) and that do not, two configurations added up.
Whole numbers: equality with the oracle."""
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
