"""The solve graph and the warp-cooperative switch on the edge games: single
games below 2^20 vertices go to the persistent solver by default, so here they
take the graph as a batch, with patches always, with the warp kernel, or padded
to more than 2^20 vertices with Odd self-loops.  Each against the oracle, in
counts, strategy and winning sets."""
import numpy as np
import pytest

import oracle
import psi
from test_edge_cases import EDGE_GAMES
from test_root_walk import paths_game, restated


def odd_leaves_even_loop():
    """Odd's first choice leads to a loop Even wins, its other one to a loop
    Odd wins: +inf until Odd's first switch, and no vertex is Even's."""
    return psi.Game.from_csr([1, 1, 1], [0, 2, 1], [0, 2, 3, 4], [1, 2, 1, 2])


def odd_leaves_even_loop_late(n=40):
    """The same at the end of a chain: v0's better choice is a chain of Odd
    vertices whose last one moves first."""
    succ = [[1, 3], [1], [2]] + [[i + 1] for i in range(3, n - 1)] + [[1, 2]]
    off = np.cumsum([0] + [len(x) for x in succ]).astype(np.int32)
    pri = np.zeros(n, np.int32)
    pri[[1, 2]] = 2, 1
    return psi.Game.from_csr(np.ones(n, np.int32), pri, off, np.array([u for x in succ for u in x], np.int32))


GAMES = {k: f for k, f in EDGE_GAMES.items() if k != "empty"}
GAMES["odd_leaves_even_loop"] = odd_leaves_even_loop
GAMES["odd_leaves_even_loop_late"] = odd_leaves_even_loop_late


def padded(g, n):
    """g and Odd self-loops of odd priority up to n vertices."""
    owner, pri, off, tgt = g.csr()
    k = n - g.n
    return psi.Game.from_csr(np.concatenate([owner, np.ones(k, np.int32)]), np.concatenate([pri, np.ones(k, np.int32)]),
                             np.concatenate([off, off[-1] + 1 + np.arange(k, dtype=np.int32)]),
                             np.concatenate([tgt, g.n + np.arange(k, dtype=np.int32)]))


def expected(g, reset=False):
    ref = oracle.Sparse(*g.csr())
    out = ref.solve(reset=reset), ref.get_strategy(), ref.get_winning(0), ref.get_winning(1)
    ref.close()
    return out


def same(got, want):
    assert got[0] == want[0]
    for x, y in zip(got[1:], want[1:]):
        assert np.array_equal(x, y)


def solved(s, reset=False):
    return s.solve(reset=reset), s.get_strategy(), s.get_winning(0), s.get_winning(1)


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(incremental=2), dict(switch_kernel=1), dict(incremental=2, graph=0),
                                dict(incremental=0, switch_kernel=1)])
@pytest.mark.parametrize("name", sorted(GAMES))
def test_graph_solves_match_the_oracle(name, kw):
    g = GAMES[name]()
    s = psi.GPUList(g, **kw)
    for reset in (False, True):
        same(solved(s, reset), expected(g, reset))
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("names", [[k] for k in sorted(GAMES)] + [
    ["all_odd", "odd_leaves_even_loop", "odd_self_loop_even"], ["all_even", "even_self_loop_odd"], sorted(GAMES)])
@pytest.mark.parametrize("graph", [0, 1])
def test_batches_match_the_oracle(names, graph):
    games = [GAMES[k]() for k in names]
    b = psi.Batch(games, graph=graph)
    for _ in range(2):
        iters, brs = b.solve()
        for k, g in enumerate(games):
            same(((iters[k], brs[k]), b.get_strategy(k), b.get_winning(k, 0), b.get_winning(k, 1)), expected(g))
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["all_odd", "all_even", "odd_leaves_even_loop", "odd_leaves_even_loop_late", "two_cycle",
                                  "cycle_forest", "odd_self_loop_even"])
def test_large_games_match_the_oracle(name):
    g = padded(GAMES[name](), (1 << 20) + 1)
    s = psi.GPUList(g)
    for reset in (False, True):
        same(solved(s, reset), expected(g, reset))
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,deg,fused", [(1000003, 14, True), (1000003, 15, False), (900000, 15, True)])
def test_dense_games_of_seven_vertices_per_thread_take_the_graph(n, deg, fused):
    """Past 933,888 vertices (152 SMs) the persistent solver, one launch, has
    games up to a mean degree of 14; the results are the same."""
    g = psi.Game.random(n, deg, deg, n, deg)
    s = psi.GPUList(g)
    s.solve()                               # (the graph is built, which counts its launches)
    before = psi.launch_count()
    got = solved(s)
    launches = psi.launch_count() - before  # of them three read the winning sets and initialise
    assert (launches < 6) == fused, launches
    w = psi.GPUList(g, switch_kernel=1)
    same(got, solved(w))
    w.close()
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("chains,cycle", [([3000, 1090], 0), ([3000, 1500], 0), ([200000, 150000, 60], 0),
                                          ([5], 400000), ([170000, 100], 150000), ([40] * 9000, 7)])
def test_walks_cut_short_in_numbers(chains, cycle):
    """More of them than one block takes (4,096) and than the grid has threads
    (155,648 on 152 SMs), in chains, on cycles and before them; in full twice,
    the second time after a switch step."""
    g = paths_game(chains, len(chains) + cycle, cycle=cycle)
    _, pri, _, tgt = g.csr()
    s = psi.GPUList(g, incremental=2)
    s.init_strat()
    strat = tgt.copy()
    strat[0] = -1
    depth, top, cnt, inf = restated(strat.tolist(), pri.tolist())
    for again in range(2):
        if again:
            s.switch_strategy(1)
            s.set_strategy(strat)             # not listed: the next evaluation is a full one
        s.compute_valuation()
        d, t, c = s.get_summary()
        assert np.array_equal(s.get_infinite(), inf)
        assert np.array_equal(d, depth) and np.array_equal(t, top) and np.array_equal(c, cnt)
        assert s.unreached() == int((inf != 0).sum())
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2000, 9000, 100000])
@pytest.mark.parametrize("kw", [dict(), dict(graph=0), dict(incremental=2)])
def test_vertices_of_very_many_successors(n, kw):
    """The persistent solver keeps a vertex's number of successors in 12 bits
    and reads 4,095 and more anew: hubs about that size and far above it among
    ordinary vertices, with ties at any place of their lists."""
    rng = np.random.default_rng(n)
    size = rng.integers(1, 5, n)
    hubs = rng.choice(n, 12, replace=False)
    size[hubs] = [4093, 4094, 4095, 4096, 4097, 8191, 5, 6, 31, 33, 30000, 12000]
    off = np.concatenate(([0], np.cumsum(size))).astype(np.int32)
    g = psi.Game.from_csr(rng.integers(0, 2, n), rng.integers(0, 40, n), off, rng.integers(0, n, off[-1]))
    s = psi.GPUList(g, **kw)
    for reset in (False, True):
        same(solved(s, reset), expected(g, reset))
    s.close()
