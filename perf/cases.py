"""The work that users have this library do, as cases to be timed: one call of
run() is one pass through the public entry points (the psi package), from a
game in hand to its solution read back.

Kinds of cases:
  solve  a game resident in a solver (psi.GPUList) is solved in one call and
         its winning set and strategy are read back
  steps  the same game driven call by call through the StrategyImprovement
         interface (psi.solve_si), as a program written against the reference's
         solver classes does
  e2e    from host CSR arrays in page-locked memory: solver creation, solve,
         read-back, release (a program that solves each game once)
  batch  many games solved together (psi.Batch), every game's result read back
  serve  games submitted to a resident server (psi.Server) and drained

Families: "random" (owner uniform, priority uniform in [0, pri), out-degree
uniform in [deg_lo, deg_hi]) and "longpath" (a chain v -> v+1 plus one back-edge
per vertex, owner alternating).
"""
import math
import os
import random
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "parallel-si_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import psi  # noqa: E402


def _solve(name, n, lo, hi, pri, kind="solve", reset=False):
    return {"name": name, "kind": kind, "family": "random", "n": n, "deg_lo": lo, "deg_hi": hi, "pri": pri,
            "reset": reset}


def listed():
    return [
        # the smallest games there are (the smallest of a batch): launches and latency only
        _solve("random-100", 100, 2, 8, 100),
        # the smallest game a server is offered, at an odd size
        _solve("random-1537", 1537, 2, 5, 1537),
        # the size the reference's CPU path is quoted on
        _solve("random-10k", 10000, 2, 10, 10000),
        # a large member of a batch, odd size, in the variant that restarts Odd's strategy in every iteration
        _solve("reset-100k", 100003, 2, 8, 100003, reset=True),
        # few priorities, as games from verification have: many ties, comparisons walk the paths
        _solve("fewpri-256k", 262144, 2, 5, 8),
        # a mid-sized game, odd size
        _solve("random-1m", 1000003, 2, 5, 1000003),
        # the headline game
        _solve("random-16m", 1 << 24, 2, 5, 1 << 24),
        # the long-path game of the benchmark: deep strategy trees
        {"name": "longpath-8m", "kind": "solve", "family": "longpath", "n": 1 << 23, "pri": 1024, "reset": False},
        # a driver written against the reference's solver interface, one call per step
        _solve("steps-50k", 50000, 2, 8, 50000, kind="steps"),
        # one game from host arrays to its solution, solver made and released
        _solve("e2e-2m", 2000000, 2, 5, 2000000, kind="e2e"),
        # a batch of mixed sizes, log-uniform as in the benchmark
        {"name": "batch-256", "kind": "batch", "games": 256, "n_lo": 100, "n_hi": 200000, "deg_lo": 2, "deg_hi": 8},
        # requests that queue up at a server, sizes log-uniform
        {"name": "serve-24", "kind": "serve", "games": 24, "n_lo": 1000, "n_hi": 200000, "deg_lo": 2, "deg_hi": 8},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choice(("solve", "solve", "solve", "solve", "steps", "e2e", "batch", "serve"))
    lo, hi = rng.choice(((2, 5), (2, 8), (2, 10)))
    if kind in ("batch", "serve"):
        n_hi = _log_int(rng, 5000, 200000)
        return {"kind": kind, "games": rng.randint(16, 200) if kind == "batch" else rng.randint(6, 24),
                "n_lo": 100 if kind == "batch" else 1000, "n_hi": n_hi, "deg_lo": lo, "deg_hi": hi}
    if kind == "solve" and rng.random() < 0.25:
        return {"kind": "solve", "family": "longpath", "n": _log_int(rng, 1000, 1 << 22), "pri": 1024,
                "reset": rng.random() < 0.25}
    few = rng.random() < 0.25
    top = {"solve": 1 << 23, "steps": 400000, "e2e": 2000000}[kind]
    n = _log_int(rng, 100, 1 << 20 if few else top)
    return {"kind": kind, "family": "random", "n": n, "deg_lo": lo, "deg_hi": hi,
            "pri": rng.randint(4, 64) if few else n, "reset": kind != "e2e" and rng.random() < 0.25}


def _game(case, seed):
    if case["family"] == "longpath":
        return psi.Game.longpath(case["n"], case["pri"], seed)
    return psi.Game.random(case["n"], case["deg_lo"], case["deg_hi"], case["pri"], seed)


def _games(case, seed):
    # the sizes belong to the case, the games to the seed
    sizes = psi.batch_sizes(case["games"], case["n_lo"], case["n_hi"], case["games"])
    return [psi.Game.random(int(n), case["deg_lo"], case["deg_hi"], int(n), 1000 * seed + k)
            for k, n in enumerate(sizes)]


class State:
    """What a user's program holds: the solver, batch or server, and the
    page-locked buffers that results are read into."""


def prepare(case, seed):
    s = State()
    s.kind = case["kind"]
    if s.kind in ("solve", "steps", "e2e"):
        g = _game(case, seed)
        s.reset = case["reset"]
        s.won = psi.pinned(g.n)
        s.won[:] = -1   # past the winning set's end the buffer stays as it is
        s.strat = psi.pinned(g.n)
        if s.kind == "e2e":
            s.csr = []
            for a in g.csr():
                p = psi.pinned(a.size)
                p[:] = a
                s.csr.append(p)
        else:
            s.solver = psi.GPUList(g)
        g.close()
        return s
    s.games = _games(case, seed)
    if s.kind == "batch":
        s.batch = psi.Batch(s.games)
        s.at = np.concatenate(([0], np.cumsum([g.n for g in s.games])))
        s.won = np.full(int(s.at[-1]), -1, np.int32)
        s.strat = np.empty(int(s.at[-1]), np.int32)
    else:
        vertices = sum(g.n + 1 for g in s.games)
        edges = sum(g.m for g in s.games)
        s.server = psi.Server(vertices, edges, len(s.games))
    return s


def _solution(s, solver, counts):
    won = solver.get_winning(0, out=s.won)
    return {"counts": counts, "n_won": won.size, "won": s.won, "strategy": solver.get_strategy(out=s.strat)}


def run(s):
    if s.kind == "solve":
        return _solution(s, s.solver, s.solver.solve(reset=s.reset))
    if s.kind == "steps":
        return _solution(s, s.solver, psi.solve_si(s.solver, reset=s.reset))
    if s.kind == "e2e":
        solver = psi.GPUList.from_csr(*s.csr)
        out = _solution(s, solver, solver.solve())
        solver.close()
        return out
    if s.kind == "batch":
        iters, brs = s.batch.solve()
        n_won = np.empty(len(s.games), np.int32)
        for k in range(len(s.games)):
            a, b = s.at[k], s.at[k + 1]
            s.strat[a:b] = s.batch.get_strategy(k)
            won = s.batch.get_winning(k, 0)
            n_won[k] = won.size
            s.won[a:a + won.size] = won
        return {"iters": iters, "brs": brs, "n_won": n_won, "won": s.won, "strategy": s.strat}
    place = {s.server.submit(g): k for k, g in enumerate(s.games)}
    counts = np.zeros((len(s.games), 2), np.int32)
    strategy, infinite = [None] * len(s.games), [None] * len(s.games)
    left = len(s.games)
    while left:
        if not s.server.step():
            continue
        for t in s.server.finished():
            k = place[int(t)]
            counts[k] = s.server.status(int(t))[1:]
            strategy[k], infinite[k] = s.server.take(int(t))
            left -= 1
    return {"counts": counts, "strategy": strategy, "infinite": infinite}


def work(case):
    """The game read once (owner, priority, offset: 4 bytes each per vertex;
    successors: 4 per edge), its strategy written and the winning set (about
    half of the vertices).  Nothing on this path is floating point."""
    if case["kind"] in ("batch", "serve"):
        # the mean of a log-uniform size
        n = case["games"] * (case["n_hi"] - case["n_lo"]) / math.log(case["n_hi"] / case["n_lo"])
    else:
        n = case["n"]
    deg = 2 if case.get("family") == "longpath" else (case["deg_lo"] + case["deg_hi"]) / 2
    return {"bytes": n * (12 + 4 * deg + 6), "flops": 0}


def exact(case, seed):
    """Every output is a whole number: there is nothing computed in floating
    point to compare with 64 bits."""
    return None
