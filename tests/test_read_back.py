"""Results read into ordinary memory: by way of page-locked staging up to
16 KB, straight above, and a batch's winning sets in parts of 131,072 vertices.
The array's bytes and no others are written, whatever its size and place."""
import ctypes as C

import numpy as np
import pytest

import psi
from psi._lib import check, lib

GUARD = -77


def read(call, n, shift):
    """call(pointer) into n words at `shift` words into an array of its own."""
    a = np.full(n + shift + 40, GUARD, np.int32)
    got = call(C.c_void_p(a.ctypes.data + 4 * shift))
    assert (a[:shift] == GUARD).all() and (a[shift + n:] == GUARD).all()
    return got, a[shift:shift + n]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3, 4095, 4096, 4097, 16384, 16385, 70001])
def test_solver_results_into_ordinary_memory(n):
    rng = np.random.default_rng(n)
    off = np.concatenate(([0], np.cumsum(rng.integers(1, 4, n)))).astype(np.int32)
    g = psi.Game.from_csr(rng.integers(0, 2, n), rng.integers(0, 9, n), off, rng.integers(0, n, off[-1]))
    s = psi.GPUList(g)
    s.solve()
    want, won = psi.pinned(n), np.flatnonzero(s.get_infinite() == 1)
    s.get_strategy(out=want)
    for shift in (0, 1, 5):
        _, got = read(lambda p: check(lib.psi_get_strategy(s._h, p)), n, shift)
        assert np.array_equal(got, want)
        for cap in {0, 1, len(won), n}:
            k = C.c_int64()
            size = min(cap, len(won))
            _, ids = read(lambda p: check(lib.psi_get_winning(s._h, 0, p, cap, C.byref(k))), size, shift)
            assert k.value == len(won) and np.array_equal(ids, won[:size])
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [[1], [3, 2000, 1], [131071, 5, 131072], [131073, 300000]])
def test_batch_and_served_results(sizes):
    games = [psi.Game.random(n, 2, 5, n, 100 + n) if n > 5 else psi.Game.from_csr([n % 2] * n, [2] * n, range(n + 1), range(n))
             for n in sizes]
    b = psi.Batch(games)
    b.solve()
    srv = psi.Server(sum(sizes) + len(sizes), sum(g.m for g in games), len(games))
    tickets = [srv.submit(g) for g in games]
    srv.drain()
    for k, g in enumerate(games):
        s = psi.GPUList(g)
        s.solve()
        want, inf = s.get_strategy(), s.get_infinite()
        s.close()
        _, got = read(lambda p: check(lib.psi_batch_get_strategy(b._h, k, p)), g.n, 3)
        assert np.array_equal(got, want)
        for player, won in ((0, np.flatnonzero(inf == 1)), (1, np.flatnonzero(inf != 1))):
            cnt = C.c_int64()
            _, ids = read(lambda p: check(lib.psi_batch_get_winning(b._h, k, player, p, g.n, C.byref(cnt))), len(won), 1)
            assert cnt.value == len(won) and np.array_equal(ids, won)
        strat, infinite = srv.take(tickets[k])
        assert np.array_equal(strat, want) and np.array_equal(infinite, inf)
    b.close()
    srv.close()
