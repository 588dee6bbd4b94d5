"""What the C host layer makes of a backend call that fails: an error, never a result.  The layer is built over
a backend made for the purpose; no GPU is involved."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("failing_backend") / "libfailing.so")
    subprocess.run(["gcc", "-O1", "-fPIC", "-shared", "-std=gnu11", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "openfish_b200", "csrc"), "-o", so,
                    os.path.join(ROOT, "openfish_b200", "csrc", "openfish_api.c"),
                    os.path.join(HERE, "host_model", "failing_backend.c")], check=True)
    L = C.CDLL(so)
    L.openfish_b200_set_error_mode(1)
    L.set_openfish_log_level(0)
    L.openfish_b200_error_text.restype = C.c_char_p
    return L


@pytest.mark.parametrize("call,n", [("openfish_b200_last_decode_ms", 4), ("openfish_b200_last_decode_detail_ms", 8)])
def test_device_times_that_cannot_be_read_are_an_error(lib, call, n):
    ms = (C.c_float * 8)(*[7.0] * 8)
    some_gpubuf = C.create_string_buffer(256)
    getattr(lib, call)(some_gpubuf, ms)
    assert lib.openfish_b200_last_status() == 6 and b"the backend says no" in lib.openfish_b200_error_text()
    assert list(ms) == [0.0] * n + [7.0] * (8 - n)
