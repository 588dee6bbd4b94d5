"""Scans that run ahead of their checks: the order of their groups built for the host.  Whatever guesses are wrong
and whenever the checker gets round to a check, every row that leaves is what each timestep taken exactly gives."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("group_order") / "libgroup_order.so")
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-o", so, os.path.join(HERE, "host_model", "group_order.cpp")], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("E,S", [(6, 6), (4, 6), (4, 5), (3, 5), (2, 5), (2, 4)])
def test_every_row_that_leaves_is_right(host, E, S):
    # the kernels' groups and stages; nearly all timesteps guessed and half of them wrong, ordinary ones, none; with
    # guesses too many for a check at times
    backs, late = C.c_int(), C.c_int()
    seen = [0, 0]
    for marked, wrong, many in ((95, 50, 99), (70, 10, 99), (30, 60, 99), (5, 100, 99), (100, 0, 99), (95, 50, 2), (60, 30, 3),
                                (100, 0, 1)):
        for T in list(range(1, 3 * E + 2)) + [E * S, 257, 800]:
            for seed in range(12):
                n = host.wrong_rows(T, E, S, marked, wrong, many, 1 + seed, C.byref(backs), C.byref(late))
                assert n == 0, (marked, wrong, many, T, seed, n, backs.value)
                seen[0] += backs.value
                seen[1] += late.value
    assert seen[0] > 1000 and seen[1] > 100  # (that the scan goes back, and a check is late beside it, does occur)
