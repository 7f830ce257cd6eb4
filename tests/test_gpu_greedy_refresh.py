"""The greedy's maps counted by tiles -- the balls of few uncovered words, or
of the words covered since the last map counted off it -- against the
transform of the masks: every placed word must be the lowest one with the
highest value of the transform's map of the words that were uncovered before
it.  Cells of a million words and more, where the tile form is taken, among
them an alphabet without tile kernels of its own."""
import numpy as np
import pytest

from coldcase_gb300.lns import TransformEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,n,R", [(2, 16, 2), (3, 13, 4), (4, 11, 4), (5, 9, 2), (6, 8, 3), (8, 7, 3),
                                   (10, 6, 2), (11, 6, 3), (16, 5, 2), (9, 7, 6)])
@pytest.mark.parametrize("take", [0.02, 0.3])
def test_placements_follow_the_transform_map(covlib, q, n, R, take):
    e, ref = TransformEngine(q, n, R), TransformEngine(q, n, R)
    try:
        e.recount(np.arange(1))
        full = np.concatenate([np.arange(1, dtype=np.int64), e.greedy(4000)[0].astype(np.int64)])
        keep = full[:len(full) - max(2, int(take * len(full)))]
        e.recount(keep)
        placed, left, _, _ = e.greedy(25)
        placed = placed.astype(np.int64)
        assert len(placed) > 0
        ref.recount(keep)
        for x in placed:
            ref.gain_map()
            m = ref.map()
            assert x == int(np.argmax(m)) and m[x] > 0
            left_ref = ref.apply(np.array([x]), 1)
        assert left == left_ref == e.count(0)
        assert (e.cnt() == ref.cnt()).all()
    finally:
        e.close()
        ref.close()
