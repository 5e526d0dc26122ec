"""GPU: the tail's ranking and merge at the numbers of peaks where its form changes
-- none, one, a word of candidates and one more, the most that one CTA takes alone,
a whole chunk, several chunks -- on chosen accumulators against the oracle."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 8, 32, 33, 128, 129, 300, 1024, 1025, 2500])
@pytest.mark.parametrize("k", [7, 400])
def test_lines_of_n_peaks(cuda, n, k):
    import torch
    from opencuda_gb300.houghline import HoughLine
    w, h, det = 900, 700, math.pi / 180
    hl = HoughLine(detheta=det, threshold=10)
    g = hl.geometry(w, h)
    acc = np.zeros((g.numrho, g.numtheta), np.int32)
    rng = np.random.default_rng(n)
    rows, cols = np.meshgrid(np.arange(4, g.numrho - 4, 3), np.arange(1, g.numtheta - 1, 3),
                             indexing="ij")
    at = rng.permutation(rows.size)[:n]
    acc[rows.ravel()[at], cols.ravel()[at]] = rng.integers(11, 60, n)   # many ties
    rc, got = hl.lines_from_accumulator(torch.from_numpy(acc).cuda(), w, h, k)
    assert rc == 0
    geo = O.geom(g.numtheta, g.rho_min, g.numrho, O.ref_numrho(w, h), det, hl.getThresDis(),
                 hl.getThresAng())
    pk = O.peaks(acc, 10)
    assert len(pk) == n
    want, _, _ = O.rank_merge(acc, geo, pk, k)
    assert [l.astuple() for l in got] == want
