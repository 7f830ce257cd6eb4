"""The engine's queued commit events, one-walk candidate list and warp-level
selection against the oracle, move by move, where they can go wrong: a last
position of more than eight values (two chunks of an item), fewer items than a
warp has lanes, more codewords than shared memory holds (notes in global
memory), codes with every codeword a candidate, a fixed first codeword."""
import numpy as np
import pytest

from coldcase_gb300.engine import Pool

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cluster", [1, 8])
@pytest.mark.parametrize("q,n,R,M,moves,opt", [
    (2, 5, 1, 6, 200, {}),              # 5 items of a single value, ties everywhere
    (2, 16, 5, 24, 150, {}),            # one value a position, many positions
    (9, 4, 2, 33, 150, {}),             # eight values: one full chunk
    (10, 4, 2, 40, 150, {}),            # nine values: a chunk of eight and one of one
    (16, 3, 1, 90, 150, {}),            # fifteen values
    (12, 4, 3, 9, 150, {}),             # nearly every word has an event
    (3, 8, 7, 2, 60, {}),               # nearly the whole space in a ball
    (6, 6, 1, 4100, 120, {}),           # codewords beyond shared memory
    (4, 6, 2, 60, 200, dict(fix0=True)),
    (7, 5, 2, 70, 200, dict(stall=20, kick=5)),
    (5, 6, 2, 120, 150, dict(noise=300)),
])
def test_moves_match_oracle(covlib, q, n, R, M, moves, opt, cluster):
    from oracle.pyoracle import Oracle
    rng = np.random.default_rng(q * 1000 + n * 10 + R)
    code = rng.integers(0, q, size=(M, n)).astype(np.uint8)
    o = Oracle(q, n, R, M, seed=5, tabu=3, threads=4, **opt)
    o.init(code)
    want = o.run(moves, trace=True)
    pool = Pool(1, cluster=cluster)
    s = pool.add(q, n, R, M, code=code, seed=5, tabu=3, trace=1, trace_cap=moves, **opt)
    pool.run(moves)
    assert pool.status(s)["status"] == 0
    assert pool.trace(s).tobytes() == want.tobytes()
    assert (pool.cnt(s) == o.cnt()).all() and (pool.best(s) == o.best()).all()
    assert (pool.rng(s) == o.rng()).all() and (pool.tabu(s) == o.tabu()).all()
    pool.close()
    o.close()


def test_initialisation_of_small_and_large_slots(covlib):
    """Slots of very different sizes added and loaded in one pool (the list
    storage follows the cell): each starts from the oracle's state."""
    from oracle.pyoracle import Oracle
    rng = np.random.default_rng(3)
    cells = [(2, 4, 1, 3), (3, 11, 2, 700), (8, 7, 4, 60), (16, 2, 1, 10), (3, 3, 0, 20)]
    pool = Pool(len(cells), cluster=1)
    slots = []
    for q, n, R, M in cells:
        code = rng.integers(0, q, size=(M, n)).astype(np.uint8)
        slots.append(pool.add(q, n, R, M, code=code, seed=7))
    for s, (q, n, R, M) in zip(slots, cells):
        code = rng.integers(0, q, size=(M, n)).astype(np.uint8)
        o = Oracle(q, n, R, M, seed=9)
        o.init(code)
        pool.load(s, code=code, seed=9)
        assert (pool.cnt(s) == o.cnt()).all()
        st = pool.status(s)
        assert st["uncovered"] == o.uncovered() and st["best"] == o.best_uncovered()
        o.close()
    pool.close()


@pytest.mark.parametrize("cluster", [1, 2, 16])
def test_cluster_wide_candidates_match_oracle(covlib, cluster):
    """Codes so long that the cluster walks them together, the best code kept
    from the changed codewords alone, kicks and a first codeword held fixed
    included; moves split over launches."""
    from oracle.pyoracle import Oracle
    for q, n, R, M, opt in ((6, 6, 1, 8400, dict(kick=70, stall=3)), (8, 6, 1, 8200, dict(fix0=True)),
                            (7, 7, 2, 8193, {}), (6, 7, 1, 20011, dict(noise=200))):
        rng = np.random.default_rng(M)
        code = rng.integers(0, q, size=(M, n)).astype(np.uint8)
        o = Oracle(q, n, R, M, seed=5, tabu=3, threads=4, **opt)
        o.init(code)
        want = o.run(90, trace=True)
        pool = Pool(1, cluster=cluster)
        s = pool.add(q, n, R, M, code=code, seed=5, tabu=3, trace=1, trace_cap=90, **opt)
        for k in (1, 50, 39):
            pool.run(k)
        assert pool.status(s)["status"] == 0
        assert pool.trace(s).tobytes() == want.tobytes()
        assert (pool.best(s) == o.best()).all() and (pool.code(s) == o.code()).all()
        assert (pool.cnt(s) == o.cnt()).all() and (pool.rng(s) == o.rng()).all()
        pool.close()
        o.close()
