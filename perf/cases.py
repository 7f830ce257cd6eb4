"""The workloads by which this framework's speed is measured.

Each case is one thing a user of the package has it do, through its public
entry points: a search on one cell (coldcase_gb300.engine), many restarts in
one launch, a mix of solve requests through the server (coldcase_gb300.serve),
many short chains (cov_chain_run), the verifier on host buffers
(coldcase_gb300.verify), the distance transform and the coverage count on
device buffers (cov_mindist_dev, cov_count_dev), the transform-engine search
(coldcase_gb300.lns) and the quotient search (coldcase_gb300.sym).

listed() are fixed sizes from the smallest calls to the largest; draw() gives
further cases of the same kinds, sizes and options; prepare(), run(), work()
and exact() serve both.  Every result is a whole number or a byte.
"""
import ctypes
import math

import numpy as np
import torch

from coldcase_gb300 import lib as L
from coldcase_gb300 import verify
from coldcase_gb300.engine import Pool
from coldcase_gb300.lns import LNS, TransformEngine
from coldcase_gb300.serve import Server
from coldcase_gb300.sym import SymPool
from coldcase_gb300.workloads import ball_volume, instance_seed, uniform_code


def listed():
    return [
        # A search on a small cell, as covsearch_gpu runs it: the counters fit
        # a few SMs' caches and a move is a chain of short steps.
        dict(name="search_q4n6", kind="search", q=4, n=6, R=1, M=300, tabu=10, cluster=2, grid_help=0, wide=False,
             warm=300, moves=500),
        # The usual single search: one cell of ten million words, one
        # instance at covsearch_gpu's cluster size.
        dict(name="search_q6n9", kind="search", q=6, n=9, R=4, M=700, tabu=20, cluster=8, grid_help=0, wide=False,
             warm=300, moves=1000),
        # A small alphabet, a long word and few codewords, with the wide
        # neighbourhood (--wide) and no tabu tenure.
        dict(name="search_wide_q3n11", kind="search", q=3, n=11, R=4, M=81, tabu=0, cluster=4, grid_help=0,
             wide=True, warm=300, moves=500),
        # The headline batch: 64 restarts of one cell advanced in one launch
        # per step, loaded from host codes and read back, as a portfolio does.
        dict(name="restarts_64_q7n9", kind="restarts", q=7, n=9, R=4, M=1500, tabu=20, count=64, cluster=2,
             warm=1000, moves=500),
        # A burst of uneven solve requests through the server: admission,
        # launches over the mix, each answer checked by the verifier.
        dict(name="served_24", kind="served", count=24, mix=2027, max_words=11_000_000, min_moves=100,
             max_moves=1000),
        # Many short independent chains on a tiny cell in one call.
        dict(name="chains_256_q6n6", kind="chains", q=6, n=6, R=3, M=41, count=256, moves=500),
        # The smallest call of all: verifying a found code of a small cell
        # from host memory (distances, histogram, covering radius).
        dict(name="verify_q6n6", kind="verify", q=6, n=6, M=41, want_dist=True),
        # The distance transform of a code held on the device, over the
        # largest word space in use: a gigabyte of distances.
        dict(name="distance_q8n10", kind="distance", q=8, n=10, M=2549),
        # The coverage multiplicity of the headline cell's code.
        dict(name="count_q7n9", kind="count", q=7, n=9, R=4, M=1500),
        # A greedy code built from nothing by the transform engine (the seed
        # of a search): recount, maps and exact placements.
        dict(name="fill_q6n9", kind="fill", q=6, n=9, R=4, M=700),
        # Ruin-and-recreate rounds on a nearly covering code of the headline
        # cell.
        dict(name="rounds_q7n9", kind="rounds", q=7, n=9, R=4, M=1329, rounds=6),
        # The quotient search on its big cell, one instance with its
        # estimates over the whole GPU (as symsearch_gpu runs it).
        dict(name="quotient_q8n9", kind="quotient", q=8, n=9, R=4, M=940, cluster=16, moves=300),
    ]


def _cell(rng, qs, ns, rs, max_words, lo=1.3, hi=7.0, max_m=65535):
    """A cell (q, n, R) whose q^n words lie within a factor of three of a size
    drawn evenly on a logarithmic scale up to max_words, and a code size
    between lo and hi times the sphere-covering quotient."""
    while True:
        words = math.exp(rng.uniform(math.log(4000), math.log(max_words)))
        cells = [(q, n, R) for q in qs for n in ns for R in rs
                 if R < n - 1 and 4000 <= q ** n <= max_words and words / 3 <= q ** n <= words * 3]
        if not cells:
            continue
        q, n, R = rng.choice(cells)
        f = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        M = math.ceil(f * q ** n / ball_volume(q, n, R))
        if 8 <= M <= max_m:
            return q, n, R, M


def draw(rng):
    kind = rng.choice(["search", "search", "restarts", "served", "chains", "verify", "distance", "distance", "count",
                       "count", "fill", "rounds", "quotient"])
    if kind == "search":
        q, n, R, M = _cell(rng, range(3, 9), range(6, 12), range(1, 5), 50_000_000, max_m=20000)
        big = q ** n >= 1 << 20
        return dict(kind=kind, q=q, n=n, R=R, M=M, tabu=rng.choice([0, 10, 20]),
                    cluster=rng.choice([8, 16]) if big else rng.choice([1, 2, 4]),
                    grid_help=rng.choice([0, 64]) if big else 0, wide=not big and rng.random() < 0.4,
                    warm=rng.randint(100, 300), moves=rng.randint(200, 1000))
    if kind == "restarts":
        q, n, R, M = _cell(rng, range(5, 8), range(7, 10), range(2, 5), 41_000_000, lo=2.0, max_m=6000)
        return dict(kind=kind, q=q, n=n, R=R, M=M, tabu=20, count=rng.randint(24, 64), cluster=2,
                    warm=rng.randint(200, 600), moves=rng.randint(100, 400))
    if kind == "served":
        return dict(kind=kind, count=rng.randint(8, 24), mix=rng.randint(1, 10 ** 6),
                    max_words=rng.randint(300_000, 11_000_000), min_moves=50, max_moves=rng.randint(200, 1000))
    if kind == "chains":
        q, n, R, M = _cell(rng, range(4, 8), range(5, 9), range(2, 5), 300_000, lo=1.5, hi=4.0, max_m=400)
        return dict(kind=kind, q=q, n=n, R=R, M=M, count=rng.randint(32, 256), moves=rng.randint(50, 500))
    if kind == "verify":
        q, n, R, M = _cell(rng, range(2, 11), range(4, 16), range(1, 5), 45_000_000, max_m=30000)
        return dict(kind=kind, q=q, n=n, M=M, want_dist=q ** n < 2_000_000)
    if kind == "distance":
        q, n, R, M = _cell(rng, range(2, 11), range(5, 17), range(1, 6), 1_080_000_000, max_m=30000)
        return dict(kind=kind, q=q, n=n, M=M)
    if kind == "count":
        q, n, R, M = _cell(rng, range(2, 11), range(5, 17), range(1, 6), 300_000_000, max_m=30000)
        return dict(kind=kind, q=q, n=n, R=R, M=M)
    if kind == "fill":
        q, n, R, M = _cell(rng, range(3, 9), range(6, 12), range(2, 5), 11_000_000, lo=3.5, hi=6.0, max_m=800)
        return dict(kind=kind, q=q, n=n, R=R, M=M)
    if kind == "rounds":
        q, n, R, M = _cell(rng, range(3, 9), range(6, 12), range(2, 5), 41_000_000, lo=3.0, hi=5.5, max_m=1400)
        return dict(kind=kind, q=q, n=n, R=R, M=M, rounds=rng.randint(3, 8))
    q, n, R, M = _cell(rng, range(4, 9), range(7, 10), range(2, 5), 140_000_000, lo=1.1, hi=3.0, max_m=3000)
    return dict(kind="quotient", q=q, n=n, R=R, M=max(M, 2 * q), cluster=rng.choice([8, 16]),
                moves=rng.randint(50, 300))


def _requests(case, seed):
    """`count` uneven solve requests: q in 5..7, n in 6..9, R in 1..4 at 1.3
    times the sphere-covering quotient, move budgets spread over their
    logarithm.  The mix is the case's; the codes and streams are the seed's."""
    rng = np.random.default_rng(case["mix"])
    out = []
    while len(out) < case["count"]:
        q, n, R = int(rng.integers(5, 8)), int(rng.integers(6, 10)), int(rng.integers(1, 5))
        M = math.ceil(1.3 * q ** n / ball_volume(q, n, R))
        if q ** n > case["max_words"] or M > 65535:
            continue
        moves = int(round(math.exp(rng.uniform(math.log(case["min_moves"]), math.log(case["max_moves"])))))
        s = instance_seed(seed, len(out))
        out.append(dict(id=len(out), q=q, n=n, R=R, M=M, seed=s, moves=moves, arrival=0.0,
                        code=uniform_code(q, n, M, s)))
    return out


def _warmed(pool, slots, moves):
    """Codes of a search under way: `moves` moves past a random start."""
    pool.run(moves)
    return [pool.code(s) for s in slots]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "served":
        return dict(case=case, server=Server(max_slots=case["count"], chunk=256), requests=_requests(case, seed))
    q, n, M = case["q"], case["n"], case["M"]
    if kind in ("search", "restarts"):
        count = case.get("count", 1)
        pool = Pool(count, cluster=case["cluster"], budget_s=60.0)
        if case.get("grid_help"):
            pool.set_param("grid_help", case["grid_help"])
        seeds = [instance_seed(seed, i) for i in range(count)]
        slots = [pool.add(q, n, case["R"], M, code=uniform_code(q, n, M, s), seed=s, tabu=case["tabu"],
                          wide=case.get("wide", False)) for s in seeds]
        return dict(case=case, pool=pool, slots=slots, seeds=seeds, codes=_warmed(pool, slots, case["warm"]))
    if kind == "chains":
        rows = np.zeros((case["count"], M, 16), dtype=np.uint8)
        for i in range(case["count"]):
            rows[i, :, :n] = uniform_code(q, n, M, instance_seed(seed, i))
        return dict(case=case, rows=rows, seed=seed % (1 << 31))
    if kind == "fill":
        return dict(case=case, engine=TransformEngine(q, n, case["R"]),
                    start=np.sort(np.random.default_rng(seed).choice(q ** n, size=2, replace=False)))
    if kind == "rounds":
        e = LNS(q, n, case["R"], seed=seed)
        e.load(np.random.default_rng(seed).choice(q ** n, size=3, replace=False))
        e.recreate(M)
        if e.uncov == 0:                 # the greedy covers below M: work at 95 % of its size
            e.ruin(len(e.code) - int(0.95 * len(e.code)), "soft")
        return dict(case=case, search=e, code=e.code.copy(), seed=seed)
    if kind == "quotient":
        return dict(case=case, pool=SymPool(1, cluster=case["cluster"], budget_s=60.0, grid_eval=True), seed=seed)
    code = uniform_code(q, n, M, seed)
    if kind == "verify":
        return dict(case=case, code=code)
    N = q ** n
    state = dict(case=case, code=torch.from_numpy(code).cuda())
    if kind == "distance":
        state["out"] = torch.empty(N, dtype=torch.uint8, device="cuda")
    else:
        state["out"] = torch.empty(N + (N & 1), dtype=torch.int16, device="cuda")   # whole 32-bit pairs
    return state


def _search_pass(st):
    """Load host codes, advance every instance, read codes and statuses back:
    one step of a program that keeps its codes between launches."""
    c, pool = st["case"], st["pool"]
    for s, code, seed in zip(st["slots"], st["codes"], st["seeds"]):
        pool.load(s, code, seed=seed)
    pool.run(c["moves"])
    stat = pool.status_all(len(st["slots"]))
    scalars = np.array([[d[k] for k in ("it", "uncovered", "best", "kicks", "status", "finished")] for d in stat],
                       dtype=np.int64)
    return dict(scalars=scalars, code=np.stack([pool.code(s) for s in st["slots"]]),
                best=np.stack([pool.best(s) for s in st["slots"]]),
                rng=np.stack([pool.rng(s) for s in st["slots"]]).view(np.int64))


def _served_pass(st):
    srv = st["server"]
    srv.done.clear()
    srv.serve(st["requests"])
    done = sorted(srv.done, key=lambda r: r["id"])
    return dict(results=np.array([[r["result"][k] for k in ("uncovered", "iters", "kicks")] for r in done],
                                 dtype=np.int64),
                codes=np.concatenate([r["best"].ravel() for r in done]))


def _chains_pass(st):
    c, rows = st["case"], st["rows"]
    k = c["count"]
    best = np.zeros_like(rows)
    best_u, solved, iters = np.zeros(k, np.int32), np.zeros(k, np.int32), np.zeros(k, np.int64)
    i32, i64 = ctypes.POINTER(ctypes.c_int32), ctypes.POINTER(ctypes.c_int64)
    L.check(L.load().cov_chain_run(c["q"], c["n"], c["R"], c["M"], k, c["moves"], st["seed"], 0, L.u8ptr(rows),
                                   L.u8ptr(best), best_u.ctypes.data_as(i32), solved.ctypes.data_as(i32),
                                   iters.ctypes.data_as(i64)), "cov_chain_run")
    return dict(best=best, best_u=best_u, solved=solved, iters=iters)


def _quotient_pass(st):
    c, pool = st["case"], st["pool"]
    s = pool.add(c["q"], c["n"], c["R"], c["M"], seed=st["seed"])
    pool.run(c["moves"])
    d = pool.status(s)
    out = dict(rep=pool.rep(s), best=pool.best(s), rng=pool.rng(s).view(np.int64),
               scalars=np.array([d[k] for k in ("it", "uncovered", "best", "kicks", "status")], dtype=np.int64))
    pool.remove(s)
    return out


def _filled(words, k):
    """The words (fewer than k once they cover) in an array of k."""
    out = np.full(k, -1, dtype=np.int64)
    out[:len(words)] = words
    return out


def _rounds_pass(st):
    c, e = st["case"], st["search"]
    e.rng = np.random.default_rng(st["seed"])
    e.load(st["code"])
    e.lns(len(st["code"]), budget_s=60.0, kmin=8, max_rounds=c["rounds"])
    k = len(st["code"])
    return dict(code=_filled(e.code, k), uncovered=int(e.uncov), best=_filled(e.best_code, k),
                best_uncovered=int(e.best_uncov))


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind in ("search", "restarts"):
        return _search_pass(state)
    if kind == "served":
        return _served_pass(state)
    if kind == "chains":
        return _chains_pass(state)
    if kind == "quotient":
        return _quotient_pass(state)
    if kind == "rounds":
        return _rounds_pass(state)
    if kind == "fill":
        e = state["engine"]
        e.recount(state["start"])
        placed, uncovered, _, _ = e.greedy(c["M"])
        return dict(placed=_filled(placed, c["M"]), uncovered=uncovered)
    if kind == "verify":
        dist, hist, radius = verify.mindist(state["code"], c["q"], c["n"], want_dist=c["want_dist"])
        return dict(dist=dist, hist=hist, radius=radius)
    stream, code, out = torch.cuda.current_stream().cuda_stream, state["code"], state["out"]
    if kind == "distance":
        L.check(L.load().cov_mindist_dev(c["q"], c["n"], code.data_ptr(), c["M"], out.data_ptr(), stream),
                "cov_mindist_dev")
        return out
    L.check(L.load().cov_count_dev(c["q"], c["n"], c["R"], code.data_ptr(), c["M"], out.data_ptr(), stream),
            "cov_count_dev")
    return out[:c["q"] ** c["n"]]


def work(case):
    """Bytes and operations one pass cannot do without: inputs once, outputs
    once, the counters that the moves and balls of the path must touch (read
    and written), and one operation per counter change or per word and axis."""
    kind = case["kind"]
    if kind == "served":
        total = dict(bytes=0.0, flops=0.0)
        for r in _requests(case, 1):
            w = _search_work(r["q"], r["n"], r["R"], r["M"], r["moves"])
            total = dict(bytes=total["bytes"] + w["bytes"], flops=total["flops"] + w["flops"])
        return total
    q, n, M = case["q"], case["n"], case["M"]
    N = q ** n
    if kind in ("search", "restarts", "chains"):
        w = _search_work(q, n, case["R"], M, case["moves"])
        return {k: v * case.get("count", 1) for k, v in w.items()}
    if kind in ("verify", "distance"):
        return dict(bytes=float(M * n + (N if case.get("want_dist", True) else 0)), flops=float(n * N))
    if kind == "count":
        R = case["R"]
        return dict(bytes=float(M * n + 2 * N), flops=float(min(M * ball_volume(q, n, R), n * (R + 1) * N)))
    ball = ball_volume(q, n, case["R"])
    if kind == "fill":
        return dict(bytes=float(2 * N + 4 * M * ball), flops=float(M * ball + n * (case["R"] + 1) * N))
    if kind == "rounds":
        k = case["rounds"] * (8 + (max(9, M // 20) - 8) // 4)   # codewords out and in
        return dict(bytes=float(2 * N + 2 * k * 4 * ball), flops=float(2 * k * ball + n * (case["R"] + 1) * N))
    # quotient: every move commits 2 S' counters and estimates some 64 candidates from 2-bit counts
    sp = q * math.comb(n - 2, case["R"]) * (q - 1) ** case["R"] / 2
    return dict(bytes=float(2 * N // q + case["moves"] * sp * (8 + 64 * 0.5)), flops=case["moves"] * sp * 2 * 66.0)


def _search_work(q, n, R, M, moves):
    sp = math.comb(n - 1, R) * (q - 1) ** R           # words a move takes out of (and into) a ball
    return dict(bytes=float(2 * q ** n + M * n * 2 + moves * (2 * sp * 4 + 8 * M)),
                flops=float(M * ball_volume(q, n, R) + moves * 4 * sp))


def exact(case, seed):
    """The transform's and the count's outputs by plain torch in 64 bits: one
    axis at a time, the least distance or the counts by distance."""
    kind = case["kind"]
    if kind not in ("verify", "distance", "count") or case["q"] ** case["n"] > 50_000_000:
        return None
    q, n = case["q"], case["n"]
    code = torch.from_numpy(uniform_code(q, n, case["M"], seed).astype(np.int64)).cuda()
    at = torch.zeros(len(code), dtype=torch.int64, device="cuda")
    for j in range(n):
        at = at * q + code[:, j]
    N = q ** n
    if kind == "count":
        R = min(case["R"], n)
        layers = [torch.zeros(N, dtype=torch.int64, device="cuda") for _ in range(R + 1)]
        layers[0].index_add_(0, at, torch.ones_like(at))
        for j in range(n):
            shape = (q ** j, q, -1)
            for d in range(R, 0, -1):
                below = layers[d - 1].view(shape)
                layers[d].view(shape).add_(below.sum(1, keepdim=True) - below)
        return sum(layers).clamp_(max=65535)
    dist = torch.full((N,), n + 1, dtype=torch.int64, device="cuda")
    dist[at] = 0
    for j in range(n):
        line = dist.view(q ** j, q, -1)
        line.copy_(torch.minimum(line, line.amin(1, keepdim=True) + 1))
    dist.clamp_(max=n + 1)
    if kind == "distance":
        return dist
    hist = torch.bincount(dist, minlength=n + 2)
    return dict(dist=dist if case["want_dist"] else None, hist=hist, radius=int(dist.max()))
