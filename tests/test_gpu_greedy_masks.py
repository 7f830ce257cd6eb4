"""The greedy on masks of uncovered words against a plain CPU greedy: blocks
of one to six digits, a word space of a single block, candidate caps down to
one, cells whose candidates outnumber the GPU's CTAs and cells with a handful;
lists of +-1 balls at once, saturated counts and repeats included; ordered
extraction across chunks."""
import itertools

import numpy as np
import pytest

from coldcase_gb300.lns import TransformEngine

pytestmark = pytest.mark.gpu


def balls(q, n, R):
    words = np.array(list(itertools.product(range(q), repeat=n)), dtype=np.int64)
    return (words[:, None, :] != words[None, :, :]).sum(2) <= R


def plain(B, code, room):
    cov = B[code].sum(0) if len(code) else np.zeros(len(B), dtype=np.int64)
    gain = (B & (cov == 0)[None, :]).sum(1)
    out = []
    while len(out) < room and (cov == 0).any():
        x = int(np.argmax(gain))
        if gain[x] <= 0:
            break
        out.append(x)
        new = B[x] & (cov == 0)
        cov = cov + B[x]
        gain = gain - B[:, new].sum(1)
    return out, int((cov == 0).sum())


@pytest.mark.parametrize("q,n,R,m0,room,cap", [
    (2, 11, 2, 3, 400, 1 << 16), (2, 4, 1, 0, 16, 1 << 16), (3, 7, 2, 2, 300, 300), (4, 5, 1, 9, 400, 1 << 16),
    (5, 4, 1, 0, 300, 50), (7, 4, 2, 1, 100, 1 << 16), (8, 4, 2, 2, 100, 1000), (9, 3, 1, 2, 200, 1 << 16),
    (13, 3, 1, 5, 300, 1 << 16), (16, 2, 1, 0, 20, 1 << 16), (11, 1, 0, 2, 9, 1 << 16), (6, 4, 4, 0, 5, 1 << 16),
    (6, 4, 0, 3, 40, 1), (5, 5, 3, 0, 60, 1)])
def test_greedy_is_the_plain_greedy(covlib, q, n, R, m0, room, cap):
    start = np.unique(np.random.default_rng(q + n + R).integers(0, q ** n, m0)) if m0 else np.zeros(0, dtype=np.int64)
    B = balls(q, n, R)
    want, unc = plain(B, start, room)
    e = TransformEngine(q, n, R)
    try:
        e.recount(start)
        placed, u, _, _ = e.greedy(room, cand_cap=cap)
        assert placed.tolist() == want and u == unc and e.count(0) == unc
        assert (e.cnt() == B[np.concatenate([start, placed]).astype(np.int64)].sum(0)).all()
        # again, after words left (the masks are made anew)
        gone = placed[::3]
        left = np.concatenate([start, np.setdiff1d(placed, gone)]).astype(np.int64)
        assert e.apply(gone, -1) == int((B[left].sum(0) == 0).sum())
        want, unc = plain(B, left, 7)
        placed, u, _, _ = e.greedy(7, cand_cap=cap)
        assert placed.tolist() == want and u == unc
    finally:
        e.close()


def test_apply_saturates_and_repeats(covlib):
    q, n, R = 5, 4, 1
    B = balls(q, n, R)
    cnt = np.zeros(q ** n, dtype=np.int64)
    e = TransformEngine(q, n, R)
    try:
        many = np.concatenate([np.full(65533, 7), np.arange(40)])
        e.recount(many)
        cnt = np.minimum(65533 * B[7] + B[np.arange(40)].sum(0), 65535)
        assert (e.cnt() == cnt).all()
        for idx, sign in ((np.full(9, 7), 1), (np.arange(0, 625, 3), 1), (np.full(5, 7), -1), (np.arange(625), -1),
                          (np.full(30, 600), -1)):
            for x in idx:
                cnt = np.clip(cnt + sign * B[x], 0, 65535)
            assert e.apply(idx, sign) == int((cnt == 0).sum())
            assert (e.cnt() == cnt).all()
    finally:
        e.close()


def test_extraction_across_chunks(covlib):
    q, n, R = 7, 6, 1
    rng = np.random.default_rng(3)
    e = TransformEngine(q, n, R)
    try:
        e.recount(rng.integers(0, q ** n, 900))
        e.gain_map()
        m = e.map()
        for thr, cap in ((1, 1 << 20), (20, 1 << 20), (20, 8192), (20, 1), (36, 5000), (38, 10), (int(m.max()), 3)):
            idx, val, found = e.map_extract(thr, cap)
            want = np.flatnonzero(m >= thr)
            assert found == len(want) and (idx == want[:cap]).all() and (val == m[want[:cap]]).all()
        words, found = e.uncovered_words(100)
        z = np.flatnonzero(e.cnt() == 0)
        assert found == len(z) and (words == z[:100]).all()
    finally:
        e.close()
