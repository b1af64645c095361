"""How the cooperative solver kernels spread vertices over threads
(csrc/spread.h), compiled for the host: no vertices at all, one, and the sizes
where the vertices per thread change."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def spread(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("cpp") / "spread")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I" + os.path.join(ROOT, "parallel-si_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "spread_main.cpp"), "-o", out], check=True)

    def call(cases):
        r = subprocess.run([out], input="".join(f"{n} {sms} {one}\n" for n, sms, one in cases), capture_output=True,
                           text=True, check=True)
        return [int(x) for x in r.stdout.split()]

    return call


def test_no_vertices(spread):
    assert spread([(0, 152, 600), (0, 152, 1024), (0, 1, 1024)]) == [128] * 3


@pytest.mark.parametrize("sms", [1, 8, 132, 152])
def test_whole_warps_that_hold_every_vertex(spread, sms):
    sizes = sorted({max(1, k * 1024 * sms + d) for k in range(0, 32) for d in (-1, 0, 1)} | {1, 2, 100, 600 * sms, 600 * sms + 1})
    for one in (600, 1024):
        for n, t in zip(sizes, spread([(n, sms, one) for n in sizes])):
            assert 128 <= t <= 1024 and t % 32 == 0, (n, t)
            each = -(-n // (1024 * sms))
            if each == 1 and n > one * sms:
                each = 2
            # one block per SM takes them all in `each` rounds
            assert t * min(sms, -(-n // t)) * each >= n, (n, t)
