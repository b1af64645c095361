"""Patches after few changes, which run in one block, that re-evaluate many
vertices: with PSI_INCR_ALWAYS there is no limit on them."""
import numpy as np
import pytest

import oracle
import psi
from lockstep import lockstep

ALWAYS = 2


def hanging(parents):
    """Even vertices 0 and n-1 start at the sink and move to n-1's self-loop of
    priority 2 in Even's first step; the Odd vertices 1 .. hang below 0 (one
    successor each, parents[i] of vertex i + 1), so they all change value."""
    n = len(parents) + 2
    succ = np.concatenate(([n - 1], parents, [n - 1])).astype(np.int32)
    owner = np.ones(n, np.int32)
    owner[[0, n - 1]] = 0
    pri = np.arange(n, dtype=np.int32) % 3
    pri[n - 1] = 2
    return psi.Game.from_csr(owner, pri, np.arange(n + 1, dtype=np.int32), succ)


def chains(count, length):
    """count chains of that length below vertex 0."""
    i = np.arange(count * length)
    return np.where(i % length == 0, 0, i)


def tree(n):
    return np.arange(n) // 3


@pytest.mark.gpu
@pytest.mark.parametrize("parents", [chains(1, 16000), chains(1, 17000), chains(40000, 1), chains(300, 90),
                                     chains(2500, 9), tree(60000)],
                         ids=["16000", "17000", "40000x1", "300x90", "2500x9", "tree"])
@pytest.mark.parametrize("graph", [0, 1])
def test_one_block_patches_have_no_limit_of_their_own(parents, graph):
    g = hanging(parents)
    s = psi.GPUList(g, incremental=ALWAYS, graph=graph)
    ref = oracle.Sparse(*g.csr())
    s.reset_times()
    if graph:
        assert s.solve() == ref.solve()
        assert np.array_equal(s.get_strategy(), ref.get_strategy())
        assert np.array_equal(s.get_infinite(), ref.get_infinite())
    else:
        lockstep(s, ref, rows=False, summary=True)
    c = s.counters()
    assert c["patches"] == c["evals"] - 1 > 0 and c["patched"] >= len(parents), c
    s.close()
    ref.close()
