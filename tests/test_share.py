"""Sharing a launch's paths among the warps of the persistent kernels
(kernel/pt_share.h): whatever the launch, a warp's slots fit its arrays."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT

SHARE_CPP = r"""
#include "pt_share.h"
extern "C" int slots(unsigned long long share, int least, int step, int cap) { return warp_slots(share, least, step, cap); }
extern "C" int chunk(unsigned long long share, int cap) { return warp_chunk(share, cap); }
"""


@pytest.fixture(scope="module")
def share(tmp_path_factory):
    d = tmp_path_factory.mktemp("share")
    src, lib = d / "s.cpp", d / "s.so"
    src.write_text(SHARE_CPP)
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-fPIC", "-shared",
                    "-I" + os.path.join(ROOT, "pathtracer_gb300", "csrc", "kernel"), "-o", str(lib), str(src)], check=True)
    so = ctypes.CDLL(str(lib))
    so.slots.argtypes = [ctypes.c_uint64] + 3 * [ctypes.c_int]
    so.chunk.argtypes = [ctypes.c_uint64, ctypes.c_int]
    return so


def _constant(source, name):
    with open(os.path.join(ROOT, "pathtracer_gb300", "csrc", "kernel", source)) as f:
        return int(f.read().split(f"constexpr int {name} = ")[1].split(";")[0])


@pytest.mark.parametrize("source,name,least,step", [("pt_persist.cu", "kPersistSlots", 32, 32),
                                                    ("pt_persist.cu", "kPersistSlots", 1, 1),
                                                    ("pt_fp64.cu", "kFp64Slots", 8, 1)])
def test_slots_fit_the_arrays(share, source, name, least, step):
    """Every share: no more slots than there are arrays for, enough for the
    share or all of them, whole steps unless all of them."""
    cap = _constant(source, name)
    for n in [*range(10001), 2**31 - 1, 2**31, 2**32 - 1, 2**32, 2**63]:
        s = share.slots(n, least, step, cap)
        assert min(least, cap) <= s <= cap, n
        assert s >= n or s == cap, n
        assert s % step == 0 or s == cap, n
        assert s == cap or s < max(n, least) + step, n


def test_claims_grow_to_their_limit(share):
    """Whole warps, never more than the limit, never fewer than for a smaller
    share, and no more than a quarter of it above the smallest claim."""
    cap = _constant("pt_persist.cu", "kPersistChunk")
    last = 0
    for n in [*range(10001), 2**31 - 1, 2**31, 2**32 - 1, 2**32, 2**63]:
        c = share.chunk(n, cap)
        assert 32 <= c <= cap and c % 32 == 0 and c >= last, n
        assert c == 32 or 4 * c <= n, n
        last = c
    assert last == cap
