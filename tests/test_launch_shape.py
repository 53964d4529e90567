"""
What a launch shape asks of the planner (csrc/hf_plan.h, compiled here for the
host): the default pair (8, 32) leaves chunk count and item length to it, every
other value in the accepted ranges is taken literally.
"""

from __future__ import annotations

import ctypes
import os
import subprocess

import pytest

from conftest import ROOT

SHIM = """
#include "hf_plan.h"
extern "C" int parts(int c, int per_sm, int nsm) { return hf::plan_parts(c, per_sm, nsm); }
extern "C" int length(long long W, int pq, int threads) { return hf::split_length(W, pq, threads); }
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, lib = d / "shim.cpp", d / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "ab-initio-md_b200", "csrc"),
                    str(src), "-o", str(lib)], check=True)
    out = ctypes.CDLL(str(lib))
    out.length.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    return out


@pytest.mark.parametrize("nsm", [1, 148])
def test_chunks(plan, nsm):
    assert plan.parts(8, 2, nsm) == 2 * nsm and plan.parts(8, 4, nsm) == 4 * nsm
    for c in [c for c in range(1, 65) if c != 8]:
        assert plan.parts(c, 2, nsm) == plan.parts(c, 4, nsm) == 2 * c * nsm


@pytest.mark.parametrize("work", [0, 1, 10 ** 5, 148 * 256 * 4 * 3, 148 * 256 * 4 * 4, 148 * 256 * 4 * 31, 10 ** 9, 2 ** 60])
def test_item_length(plan, work):
    threads = 148 * 256
    assert plan.length(work, 32, threads) == min(32, max(4, work // (4 * threads)))
    for pq in (4, 5, 31, 33, 64, 4096):         # a small launch too: 4096 is unsplit
        assert plan.length(work, pq, threads) == pq
