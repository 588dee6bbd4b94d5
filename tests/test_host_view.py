"""Which result buffers the last kernel of a decode may write itself: only what is page-locked from end
to end.  The rule on its own, built for the host, with the driver's answers made up."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("host_view") / "libhost_view.so")
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-o", so, os.path.join(HERE, "host_model", "host_view.cpp")], check=True)
    lib = C.CDLL(so)
    lib.host_writable.restype = C.c_size_t
    lib.host_writable.argtypes = [C.c_int, C.c_size_t, C.c_size_t, C.c_size_t, C.c_size_t]
    return lib


START, SIZE = 0x7f0000004000, 4 * 4096


@pytest.mark.parametrize("offset,n,direct", [(0, SIZE, True), (0, SIZE + 1, False), (8192, 8192, True), (8192, 8193, False),
                                             (SIZE - 1, 1, True), (SIZE - 1, 2, False), (SIZE, 1, False), (16, 2 ** 63, False),
                                             (-16, 32, False)])
def test_buffers_within_and_beyond_a_registration(host, offset, n, direct):
    p = START + offset
    assert host.host_writable(1, p, START, SIZE, n) == (p if direct else 0)


def test_pageable_or_unmapped_memory_is_never_written_by_the_device(host):
    assert host.host_writable(0, START, START, SIZE, 16) == 0
    assert host.host_writable(1, 0, 0, SIZE, 16) == 0
