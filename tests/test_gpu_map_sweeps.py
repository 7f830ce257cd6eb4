"""The maps over their sweep plans against the oracle's ball marking: one tile,
one, two and three strip sweeps, three to nine layers, every alphabet with its
own kernels and the generic one, tiles of a number of words that is no multiple
of four, radius 0 and the whole space; and the recount on either side of the
rule between the verifier's tiles and the transform of the word counts."""
import ctypes

import numpy as np
import pytest

from coldcase_gb300 import lib as L
from coldcase_gb300.lns import TransformEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,n,R,m", [
    (2, 3, 1, 2), (2, 16, 8, 3), (2, 15, 5, 9), (3, 1, 1, 1), (3, 12, 4, 30), (3, 9, 8, 2), (4, 4, 4, 3), (4, 9, 6, 4),
    (5, 8, 2, 90), (5, 9, 5, 5), (6, 8, 7, 3), (7, 6, 0, 50), (7, 7, 6, 4), (7, 8, 4, 20), (8, 8, 7, 3), (8, 7, 3, 40),
    (9, 6, 4, 9), (10, 6, 3, 20), (11, 5, 2, 30), (13, 5, 5, 2), (16, 4, 3, 5), (16, 5, 1, 60)])
def test_maps_equal_oracle(covlib, q, n, R, m):
    from oracle import pyoracle as po
    rng = np.random.default_rng(100 * q + 10 * n + R)
    idx = rng.integers(0, q ** n, m)
    e = TransformEngine(q, n, R)
    try:
        e.recount(idx)
        cnt = e.cnt()
        assert (cnt == po.cover_count(e.index_word(idx), q, n, R)).all()
        # the rarest multiplicity, and 0 and 1 where the marking is affordable
        values, words = np.unique(cnt, return_counts=True)
        for target in {int(values[np.argmin(words)]), 0, 1}:
            marked = np.flatnonzero(cnt == target)
            L.check(covlib.cov_lns_map(e.h, target))
            if len(marked) * float(q) ** min(n, 2 * R) > 3e8 or len(marked) > 60000:
                # too many balls for the oracle: distances at some words instead
                at = np.unique(np.concatenate([[0, q ** n - 1], rng.integers(0, q ** n, 24)]))
                got, digits = e.map()[at], e.index_word(marked)
                for x, g in zip(at, got):
                    assert int(((digits != e.index_word([x])).sum(1) <= R).sum()) == g, (target, x)
                continue
            want = np.zeros(q ** n, dtype=np.int64)
            for part in np.array_split(marked, max(1, -(-len(marked) // 60000))):
                if len(part):
                    want += po.cover_count(e.index_word(part), q, n, R)
            assert (e.map() == want).all(), target
    finally:
        e.close()


@pytest.mark.parametrize("q,n,R,m", [(6, 5, 2, 3000), (6, 5, 2, 300), (5, 5, 1, 9000), (9, 4, 0, 20000), (7, 4, 3, 5000),
                                     (3, 8, 4, 2000), (8, 5, 2, 60000)])
def test_recount_of_dense_codes(covlib, q, n, R, m):
    from oracle import pyoracle as po
    idx = np.random.default_rng(m + q).integers(0, q ** n, m)
    e = TransformEngine(q, n, R)
    try:
        e.recount(idx)
        assert (e.cnt() == po.cover_count(e.index_word(idx), q, n, R)).all()
        e.recount(idx[:1])
        assert (e.cnt() == po.cover_count(e.index_word(idx[:1]), q, n, R)).all()
    finally:
        e.close()
