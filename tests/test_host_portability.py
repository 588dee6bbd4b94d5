"""The host code is not tied to one processor: B200 boards come with aarch64 hosts as well as with x86 ones.  (There
is no compiler for another processor here: the header that differs is preprocessed as one would see it, and nothing
else may name an instruction.)"""
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "openfish_b200", "csrc")


@pytest.mark.parametrize("defines,has", [(["-D__aarch64__"], "yield"), ([], None)])
def test_the_pause_of_a_waiting_thread_on_other_processors(defines, has):
    text = subprocess.run(["g++", "-E", "-P", "-x", "c++", "-U__x86_64__", "-U__i386__", *defines, os.path.join(CSRC, "cpu_relax.h")],
                          check=True, capture_output=True, text=True).stdout
    assert "ia32" not in text and "cpu_relax" in text
    assert has is None or has in text


def test_no_other_source_names_an_instruction_of_the_host():
    for f in sorted(os.listdir(CSRC)):
        if f != "cpu_relax.h":
            with open(os.path.join(CSRC, f)) as src:
                assert not re.search(r"__builtin_ia32|_mm_\w+\(|immintrin|x86intrin", src.read()), f
