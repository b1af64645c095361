"""The step-by-step calls in orders of the caller's own: strategies set or reset
after an evaluation and switched before the next one (a switch step goes by the
last evaluation's valuations, whatever the strategies are by then)."""
import numpy as np
import pytest

import oracle
import psi
from games import make

GAMES = [("c1", 3000, 1), ("c4", 2500, 2), ("smallpri", 3000, 3), ("c3", 2000, 4)]


def random_strategy(g, rng):
    owner, _, off, tgt = g.csr()
    out = tgt[off[:-1] + rng.integers(0, 1 << 30, g.n) % (off[1:] - off[:-1])].copy()
    out[(owner == 0) & (rng.random(g.n) < 0.3)] = -1
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("incremental", [0, 1, 2])
@pytest.mark.parametrize("fam,n,seed", GAMES)
def test_switches_between_a_new_strategy_and_its_evaluation(fam, n, seed, incremental):
    g = make(fam, n, seed)
    rng = np.random.default_rng(seed)
    s, ref = psi.GPUList(g, incremental=incremental), oracle.Oracle(*g.csr())
    for x in (s, ref):
        x.init_strat()
    strategies = [random_strategy(g, rng) for _ in range(3)]
    for step in range(12):
        for x in (s, ref):
            x.compute_valuation()
        assert np.array_equal(s.get_infinite(), ref.get_infinite()), step
        if step % 4 == 1:
            for x in (s, ref):
                x.set_strategy(strategies[step // 4])
        elif step % 4 == 3:
            for x in (s, ref):
                x.reset_opponent_strategy()
        for player in (1, 0):
            assert s.switch_strategy(player) == ref.switch_strategy(player), (step, player)
            assert np.array_equal(s.get_strategy(), ref.get_strategy()), (step, player)
    s.close()
    ref.close()


@pytest.mark.gpu
def test_switches_between_a_solve_and_the_next_evaluation():
    g = make("c1", 3000, 9)
    rng = np.random.default_rng(9)
    new = random_strategy(g, rng)
    s, ref = psi.GPUList(g), oracle.Oracle(*g.csr())
    s.solve()
    ref.solve()
    for order in range(2):
        for x in (s, ref):
            x.set_strategy(new)
        for player in (1, 0):
            assert s.switch_strategy(player) == ref.switch_strategy(player)
        for step in range(3):
            for x in (s, ref):
                x.compute_valuation()
            assert np.array_equal(s.get_infinite(), ref.get_infinite())
            for player in (1, 0):
                assert s.switch_strategy(player) == ref.switch_strategy(player), (order, step, player)
                assert np.array_equal(s.get_strategy(), ref.get_strategy())
    s.close()
    ref.close()
