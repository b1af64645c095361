"""psi_solve as one persistent kernel (solve_kernels.cu) at the sizes where
its launch or its phases change: one block with everything in shared memory
below 2,000 vertices (its successors too, where they fit), blocks of 128 threads
and more above, two vertices per thread past 91,200 (152 SMs), three past
311,296, up to seven; jumps over deep chains and long cycles; and the state it
leaves for the step-by-step calls."""
import numpy as np
import pytest

import oracle
import psi
from games import make
from lockstep import lockstep
from test_root_walk import paths_game

PSI_ERR_LIMIT = 8


def _solved(s, reset=False):
    out = s.solve(reset=reset), s.get_strategy(), s.get_infinite(), s.get_solved(), s.get_winning(0)
    return out + s.get_summary()


def _same(a, b):
    assert a[0] == b[0]
    for k, (x, y) in enumerate(zip(a[1:], b[1:])):
        assert np.array_equal(x, y), f"output {k}: differ at {np.nonzero(x != y)[0][:10]}"


GAMES = [("ring10", 10, 0), ("c4", 1999, 1), ("c4", 2000, 2), ("c3", 1999, 3)]
GAMES += [("c4", n, n) for n in (20, 127, 128, 129, 1023, 1024, 1025, 2049, 19456, 19457)]
GAMES += [("smallpri", n, n) for n in (64, 1024, 1025, 30000)]
GAMES += [("c3", n, n) for n in (50, 1025, 20000)]
GAMES += [("evencyc", 3000, 5), ("cycles", 12, 3), ("cycles", 24, 4)]


@pytest.mark.gpu
@pytest.mark.parametrize("reset", [False, True])
@pytest.mark.parametrize("fam,n,seed", GAMES)
def test_solve_matches_the_oracle(fam, n, seed, reset):
    g = make(fam, n, seed)
    ref = oracle.Sparse(*g.csr())
    s = psi.GPUList(g)
    for _ in range(2):                        # a second solve starts afresh
        assert s.solve(reset=reset) == ref.solve(reset=reset)
        assert np.array_equal(s.get_strategy(), ref.get_strategy())
        assert np.array_equal(s.get_infinite(), ref.get_infinite())
        assert np.array_equal(s.get_winning(0), ref.get_winning(0))
    s.close()
    ref.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,deg", [(1, 0), (2, 1), (65, 64), (1500, 40), (1999, 45)])
def test_small_games_of_any_degree(n, deg):
    """Up to 1,999 vertices with few or many successors (past what shared
    memory holds), self-loops and repeated successors among them."""
    rng = np.random.default_rng(n)
    size = rng.integers(1, deg + 2, n)
    off = np.concatenate(([0], np.cumsum(size))).astype(np.int32)
    g = psi.Game.from_csr(rng.integers(0, 2, n), rng.integers(0, 30, n), off, rng.integers(0, n, off[-1]))
    ref = oracle.Sparse(*g.csr())
    s = psi.GPUList(g)
    for reset in (False, True):
        assert s.solve(reset=reset) == ref.solve(reset=reset)
        assert np.array_equal(s.get_strategy(), ref.get_strategy())
        assert np.array_equal(s.get_infinite(), ref.get_infinite())
    s.close()
    ref.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,pri", [(91200, 91200), (91201, 12), (155648, 155648), (155649, 9), (311296, 9),
                                   (311297, 311297), (778241, 778241), ((1 << 20) - 1, 1 << 20)])
def test_solve_matches_the_graph_loop(n, pri):
    """Against the same game through the graph (the warp-cooperative switch
    selects it), which other tests hold to the oracle at these sizes."""
    g = psi.Game.random(n, 2, 5, pri, n)
    a, b = psi.GPUList(g), psi.GPUList(g, switch_kernel=1)
    _same(_solved(a), _solved(b))
    a.close()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("chains,cycle", [
    ([1], 0), ([64], 0), ([65], 0), ([3000, 500], 0), ([0xFFFE], 0), ([0xFFFF], 0), ([70000], 0), ([100000] * 4, 0),
    ([5], 1), ([100], 2), ([900], 63), ([900], 64), ([30], 4097), ([5000] * 40, 3), ([100], 200000),
])
def test_deep_chains_and_long_cycles(chains, cycle):
    g = paths_game(chains, 7 * len(chains) + cycle, cycle=cycle)
    a, b = psi.GPUList(g), psi.GPUList(g, graph=0)
    _same(_solved(a), _solved(b))
    a.close()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cap", [1, 2, 5, 9])
@pytest.mark.parametrize("reset", [0, 1])
def test_steps_after_a_capped_solve(cap, reset):
    """A solve stopped by its evaluation cap leaves a state that the
    step-by-step calls go on from, as after the host-driven loop."""
    import ctypes as C

    from psi._lib import lib
    g = make("c1", 3000, 17)
    a, b = psi.GPUList(g), psi.GPUList(g, graph=0)
    for s in (a, b):
        it, br = C.c_int32(), C.c_int32()
        assert lib.psi_solve(s._h, reset, C.byref(it), C.byref(br), cap) == PSI_ERR_LIMIT
    for step in range(4):
        for s in (a, b):
            if step:
                s.compute_valuation()
        for p in (1, 0):
            a.mark_solved(p)
            b.mark_solved(p)
            assert a.switch_strategy(p) == b.switch_strategy(p)
        assert np.array_equal(a.get_strategy(), b.get_strategy())
        assert np.array_equal(a.get_infinite(), b.get_infinite())
        assert np.array_equal(a.get_solved(), b.get_solved())
    a.close()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1 << 20, 933_888 + 300_001, 6_000_001])
def test_claimed_switches_match_strided_ones(n):
    """Odd owns seven of eight vertices, so the first switch lists just under and
    over the entries (933,888 on 152 SMs) past which a warp claims more than
    two chunks of the list, and past those where it claims sixteen; few
    priorities, so that some walk.  The warp kernel deals by a fixed stride."""
    rng = np.random.default_rng(n)
    off = np.concatenate(([0], np.cumsum(rng.integers(1, 4, n)))).astype(np.int32)
    g = psi.Game.from_csr((rng.integers(0, 8, n) > 0).astype(np.int32), rng.integers(0, 50, n).astype(np.int32), off,
                          rng.integers(0, n, off[-1]).astype(np.int32))
    a, b = psi.GPUList(g), psi.GPUList(g, switch_kernel=1)
    _same(_solved(a), _solved(b))
    a.close()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 2])   # the persistent solver; the graph (PSI_INCR_ALWAYS)
@pytest.mark.parametrize("deg", [5, 31, 32, 33, 90])
def test_ties_at_any_place_of_a_list(deg, mode):
    """Ties among the first 32 successors are remembered, later ones asked for
    again: lists of up to deg successors, repeated ones among them, with four
    priorities, so that most best keys are shared."""
    rng = np.random.default_rng(deg)
    n = 2300
    size = rng.integers(max(1, deg - 4), deg + 1, n)
    off = np.concatenate(([0], np.cumsum(size))).astype(np.int32)
    # successors near the end of the order make long common paths
    tgt = np.minimum(n - 1, rng.integers(0, n, off[-1]) | rng.integers(0, n, off[-1])).astype(np.int32)
    g = psi.Game.from_csr(rng.integers(0, 2, n), rng.integers(0, 4, n), off, tgt)
    ref = oracle.Sparse(*g.csr())
    s = psi.GPUList(g, incremental=mode)
    for reset in (False, True):
        assert s.solve(reset=reset) == ref.solve(reset=reset)
        assert np.array_equal(s.get_strategy(), ref.get_strategy())
        assert np.array_equal(s.get_infinite(), ref.get_infinite())
    lockstep(s, ref, rows=False)              # and the number of strict improvements of every step
    s.close()
    ref.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,pri", [(20000, 2), (100000, 6), (300000, 4), (300000, 60)])
def test_landmarks_come_and_go(n, pri):
    """The graph's evaluations write landmark records only after a switch step
    that walked more than n / 2 steps (n / 8 with them) or far from one vertex:
    games with few priorities cross both ways.  Against the persistent solver,
    whose comparisons step; in full every time and with patches in between."""
    g = psi.Game.random(n, 2, 5, pri, n + pri)
    ref = psi.GPUList(g)
    for kw in (dict(incremental=2), dict(incremental=0, switch_kernel=1), dict(incremental=2, graph=0)):
        s = psi.GPUList(g, **kw)
        for _ in range(2):
            _same(_solved(s), _solved(ref))
        s.close()
    ref.close()
