"""The full evaluation's walks (root_kernels.cu), and its jumps in one launch for
games below 2^20 vertices (solve_kernels.cu), at the sizes where they change path: walks that end just before, at and after the step cap of 128 (longer
ones go through pointer jumping, in one block up to 4,096 of them, over the
grid above), cycles around the cap, paths longer than the 16-bit depth of a
path record.  Checked against a plain restatement over the same strategy."""
import numpy as np
import pytest

import oracle
import psi
from lockstep import lockstep

CAP = 128
DEEP = 0xFFFF


def paths_game(chains, seed, pri_hi=6, cycle=0):
    """Odd chains of the given lengths (one successor each) that hang off the
    Even vertex 0 (strategy: the sink) or, with cycle > 0, off a cycle of that
    many Odd vertices; ids shuffled, few priorities (so tops are shared)."""
    rng = np.random.default_rng(seed)
    succ = [0]                                  # Even vertex 0: a self-loop it does not take at first
    cyc0 = len(succ)
    succ += [cyc0 + (i + 1) % cycle for i in range(cycle)]
    for length in chains:
        at = cyc0 + int(rng.integers(cycle)) if cycle else 0
        for _ in range(length):
            succ.append(at)
            at = len(succ) - 1
    n = len(succ)
    perm = np.concatenate(([0], 1 + rng.permutation(n - 1)))
    tgt = np.empty(n, np.int32)
    tgt[perm] = perm[np.array(succ)]
    owner = np.ones(n, np.int32)
    owner[0] = 0
    pri = rng.integers(0, pri_hi, n).astype(np.int32)
    return psi.Game.from_csr(owner, pri, np.arange(n + 1, dtype=np.int32), tgt)


def restated(strat, pri):
    """(depth, top priority, its count, infinite flag) per vertex of a strategy."""
    n = len(strat)
    depth, top, cnt, inf = np.zeros(n, np.int32), np.full(n, -1, np.int32), np.zeros(n, np.int32), np.zeros(n, np.int32)
    state = np.zeros(n, np.int8)                # 1 on the current walk, 2 done
    for v0 in range(n):
        path, v = [], v0
        while v >= 0 and state[v] == 0:
            state[v] = 1
            path.append(v)
            v = strat[v]
        if v >= 0 and state[v] == 1:            # a new cycle
            k = path.index(v)
            val = 1 if max(pri[u] for u in path[k:]) % 2 == 0 else -1
            inf[path[k:]] = val
            state[path[k:]] = 2
            path = path[:k]
        for u in reversed(path):
            t = strat[u]
            state[u] = 2
            if t >= 0 and inf[t]:
                inf[u] = inf[t]
                continue
            depth[u] = 1 + (depth[t] if t >= 0 else 0)
            m, c = (top[t], cnt[t]) if t >= 0 else (-1, 0)
            top[u], cnt[u] = (pri[u], 1) if pri[u] > m else (m, c + (pri[u] == m))
    return depth, top, cnt, inf


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 2])   # jumps in one launch (PSI_INCR_OFF); walks (PSI_INCR_ALWAYS, first evaluation)
@pytest.mark.parametrize("chains,cycle", [
    ([1], 0), ([2, 3], 0), ([CAP - 2], 0), ([CAP - 1], 0), ([CAP], 0), ([CAP + 1, CAP + 2], 0), ([4 * CAP + 3] * 3, 0),
    ([4500, 4200, 70], 0), ([DEEP - 1, 40], 0), ([DEEP, 3], 0), ([DEEP + 1, 900], 0), ([70000], 0),
    ([1, 5], 1), ([40], 2), ([CAP], CAP - 1), ([CAP + 1], CAP), ([3], CAP + 1), ([60, 300], 1000), ([9], 5000),
    ([5000], 3), ([20000, 600], 4097),
])
def test_walks_match_a_plain_restatement(chains, cycle, mode):
    g = paths_game(chains, len(chains) + cycle, cycle=cycle)
    _, pri, _, tgt = g.csr()
    s = psi.GPUList(g, incremental=mode)
    s.init_strat()
    s.compute_valuation()
    strat = tgt.copy()
    strat[0] = -1
    depth, top, cnt, inf = restated(strat.tolist(), pri.tolist())
    d, t, c = s.get_summary()
    assert np.array_equal(s.get_infinite(), inf)
    assert np.array_equal(d, depth) and np.array_equal(t, top) and np.array_equal(c, cnt)
    assert s.unreached() == int((inf != 0).sum())
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("length", [300, DEEP - 2, DEEP + 5])
@pytest.mark.parametrize("incremental", [0, 2])
def test_comparisons_on_deep_paths_match_the_oracle(length, incremental):
    """Two chains of equal length and equal summaries, told apart only by a
    walk from their heads; Odd vertices choose between the heads and an Even
    vertex may close a cycle later."""
    n = 2 * length + 6
    a, b = 2, 2 + length                        # the chains' last vertices (they leave for Even vertices 0, 1)
    owner = np.ones(n, np.int32)
    owner[[0, 1, n - 1]] = 0
    pri = np.tile(np.array([4, 1, 2, 4, 3], np.int32), n // 5 + 1)[:n].copy()
    pri[[0, 1]] = 2
    pri[a:a + length] = pri[b:b + length]
    pri[a + length // 2], pri[b + length // 2] = 0, 3
    succ = [[n - 1], [n - 1]] + [[0]] + list([i - 1] for i in range(a + 1, b)) + [[1]]
    succ += [[i - 1] for i in range(b + 1, b + length)]
    heads = [b - 1, b + length - 1]
    succ += [heads, heads[::-1], [heads[1], heads[0], 0], [n - 1, heads[0]]]
    off = np.cumsum([0] + [len(x) for x in succ]).astype(np.int32)
    g = psi.Game.from_csr(owner, pri, off, np.array([u for x in succ for u in x], np.int32))
    gpu = psi.GPUList(g, incremental=incremental)
    ref = oracle.Sparse(*g.csr())
    lockstep(gpu, ref, rows=False, summary=True)
    gpu.close()
    ref.close()


def comb_game(pairs, trunk, pad, seed):
    """A trunk (a chain of Odd vertices to Even vertex 0) and pairs of equally
    long chains that leave it at random vertices; an Odd vertex per pair chooses
    between the two heads.  The trunk carries the top priorities, so the heads
    tie and are told apart below the vertices where their chains meet the
    trunk, hundreds of vertices apart.  Padded with Odd self-loops."""
    rng = np.random.default_rng(seed)
    succ, pri = [[0]], [2]
    for i in range(trunk):
        succ.append([len(succ) - 1 if i else 0])
        pri.append(int(rng.integers(40, 64)))
    for _ in range(pairs):
        length, heads = int(rng.integers(1, 260)), []
        at = int(rng.integers(trunk // 2, trunk)) + 1
        for k in range(2):
            prev = at if k == 0 or rng.random() < 0.5 else int(rng.integers(trunk // 2, trunk)) + 1
            for _ in range(length):
                succ.append([prev])
                pri.append(int(rng.integers(0, 30)))
                prev = len(succ) - 1
            heads.append(prev)
        if rng.random() < 0.3:      # the same private priorities: a tie to the end
            n = len(succ)
            pri[n - length:n] = pri[n - 2 * length:n - length]
        succ.append(heads if rng.random() < 0.5 else heads[::-1])
        pri.append(int(rng.integers(0, 30)))
    size = np.array([len(x) for x in succ] + [1] * pad, np.int64)
    n = len(size)
    tgt = np.concatenate([np.array([u for x in succ for u in x]), np.arange(len(succ), n)]).astype(np.int32)
    owner = np.ones(n, np.int32)
    owner[0] = 0
    pri = np.concatenate([pri, np.ones(pad)]).astype(np.int32)
    return psi.Game.from_csr(owner, pri, np.concatenate(([0], np.cumsum(size))).astype(np.int32), tgt)


@pytest.mark.gpu
@pytest.mark.parametrize("trunk", [70, 700, 4000])
@pytest.mark.parametrize("pad,incremental", [(0, 0), (0, 2), (1 << 20, 0), (1 << 20, 1)])
def test_ties_far_from_where_the_paths_meet(trunk, pad, incremental):
    """Small games compare on the jumps' records, larger ones along landmarks
    (with patches, whose vertices have none, in between)."""
    g = comb_game(400, trunk, pad, trunk + incremental)
    gpu = psi.GPUList(g, incremental=incremental)
    ref = oracle.Sparse(*g.csr())
    lockstep(gpu, ref, rows=False, summary=True)
    strat = ref.get_strategy()
    gpu.solve()
    assert np.array_equal(gpu.get_strategy(), strat)
    gpu.close()
    ref.close()
