"""The library's decisions that need no GPU (csrc/rules.h), compiled for the host."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = """
#include "rules.h"
extern "C" int in_place(int type, int where, int device) { return aldic::memory_in_place(type, where, device); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "2d_aldic_b200", "csrc"),
                    str(d / "shim.cpp"), "-o", str(d / "rules.so")], check=True)
    return C.CDLL(str(d / "rules.so"))


@pytest.mark.parametrize("device", [0, 1, 7])
def test_only_its_own_memory_is_used_in_place(rules, device):
    host, pinned, dev, managed = 0, 1, 2, 3       # cudaMemoryType
    for where in range(-2, 8):                    # -2, -1: of no device
        assert not rules.in_place(host, where, device)
        assert not rules.in_place(pinned, where, device)
        assert rules.in_place(dev, where, device) == (where == device)
        assert rules.in_place(managed, where, device)
