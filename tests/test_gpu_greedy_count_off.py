"""Greedy maps counted off the last map: with a candidate or two kept a
refresh, nearly every placement takes a new map, and in these cells (some two
million words or more, most of them uncovered, a few hundred newly covered
between two maps) it comes from the words covered since.  Every placed word is
the lowest one with the highest value of the transform's map."""
import numpy as np
import pytest

from coldcase_gb300.lns import TransformEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,n,R", [(8, 7, 2), (4, 11, 2), (3, 14, 3), (12, 6, 2), (7, 8, 3), (5, 10, 1), (16, 6, 1)])
@pytest.mark.parametrize("cand_cap", [1, 2])
def test_placements_follow_the_transform_map(covlib, q, n, R, cand_cap):
    e, ref = TransformEngine(q, n, R), TransformEngine(q, n, R)
    try:
        start = np.random.default_rng(q * n + R).integers(0, q ** n, 40)
        e.recount(start)
        placed, left, refreshes, _ = e.greedy(12, cand_cap=cand_cap)
        assert len(placed) == 12 and refreshes >= 4 and left > 65536
        ref.recount(start)
        for x in placed.astype(np.int64):
            ref.gain_map()
            m = ref.map()
            assert x == int(np.argmax(m)) and m[x] > 0
            left_ref = ref.apply(np.array([x]), 1)
        assert left == left_ref == e.count(0)
        assert (e.cnt() == ref.cnt()).all()
    finally:
        e.close()
        ref.close()
