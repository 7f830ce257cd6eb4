"""A quotient-search instance on the whole GPU against the oracle, move by
move: kicks of several orbits, a candidate cap (sampled subsets), more moves
than one launch takes, a sample longer than a batch of draws, and a deadline
between two orbit placements or two moves with the run resumed."""
import pytest

from coldcase_gb300.sym import SymPool

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,n,R,M,cand,kick,stall,moves", [
    (6, 8, 4, 168, 7, 0, 15, 300), (5, 6, 2, 100, 3, 1, 25, 2500), (3, 9, 2, 150, 50, 4, 40, 1200),
    (2, 10, 2, 40, 100000, 2, 30, 1025), (4, 6, 1, 200, 100000, 2, 10, 700), (8, 5, 2, 800, 100000, 2, 50, 200),
    (9, 4, 1, 300, 100000, 3, 20, 300)])
def test_grid_equals_oracle(covlib, q, n, R, M, cand, kick, stall, moves):
    from oracle.pyoracle import SymOracle
    o = SymOracle(q, n, R, M, seed=5, kick=kick, stall=stall, cand=cand)
    o.init()
    otr = o.run(moves, trace=True)
    with SymPool(1, cluster=2, grid_eval=True) as pool:
        s = pool.add(q, n, R, M, seed=5, kick=kick, stall=stall, cand=cand, trace=1, trace_cap=moves)
        pool.run(moves)
        assert pool.status(s)["status"] == 0
        gtr = pool.trace(s)
        assert len(gtr) == len(otr) and gtr.tobytes() == otr.tobytes()
        assert (pool.cnt(s) == o.cnt()).all() and (pool.best(s) == o.best()).all()
        assert (pool.rng(s) == o.rng()).all()


def test_grid_timeout_resume_keeps_trajectory(covlib):
    from oracle.pyoracle import SymOracle
    q, n, R, M, moves = 6, 8, 4, 168, 60
    o = SymOracle(q, n, R, M, seed=3)
    o.init()
    otr = o.run(moves, trace=True)
    with SymPool(1, cluster=2, budget_s=2e-5, grid_eval=True) as pool:
        s = pool.add(q, n, R, M, seed=3, trace=1, trace_cap=moves)
        stops = 0
        for _ in range(100000):
            st = pool.status(s)
            if st["status"] == -4:
                stops += 1
                pool.resume(s)
                if stops == 40:
                    pool.lib.cov_sym_set_budget(pool.h, 30.0)
            elif st["it"] >= moves or st["finished"]:
                break
            assert pool.status(s)["status"] == 0
            pool.run(moves - st["it"])
        assert stops > 0
        assert pool.trace(s).tobytes() == otr.tobytes() and (pool.cnt(s) == o.cnt()).all()
