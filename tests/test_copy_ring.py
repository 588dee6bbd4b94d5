"""The copy warp of the scans and of the beam search, its order of waits and copies built for the host: a
block must not end while a copy into its shared memory is under way, whenever it gives up."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("copy_ring") / "libcopy_ring.so")
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-o", so, os.path.join(HERE, "host_model", "copy_ring.cpp")], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("ring", [2, 4, 6])
def test_no_copy_is_under_way_when_the_copy_warp_ends(host, ring):
    # fewer groups than stages (nothing is ever waited for on the way), exactly as many, more; giving up
    # before any group, between groups, and after the last has been issued
    for groups in range(1, 4 * ring + 2):
        for stop in range(groups + 1):
            assert host.copies_left(groups, ring, stop) == 0, (groups, stop)
