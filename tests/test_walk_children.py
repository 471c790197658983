"""The rule that puts a walk step's node pairs into the next frontier
(csrc/walk_children.h, compiled here for the host): whatever part of a group of
children lies below the buffer's end is written, and nothing beyond it, for every
decision and every place of the end in or beside the group."""

from __future__ import annotations

import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from jaccpot_b200 import build

HEADER = Path(__file__).resolve().parent.parent / "jaccpot_b200" / "csrc" / "walk_children.h"
SELF, FAR, NEAR, SPLIT_A, SPLIT_B, NONE = 1, 2, 3, 4, 5, 0
LEFT, RIGHT = np.array([1, 3, 5], np.int32), np.array([2, 4, 6], np.int32)


@pytest.fixture(scope="module")
def fn(tmp_path_factory):
    d = tmp_path_factory.mktemp("walk")
    (d / "shim.cpp").write_text(f'''#include "{HEADER}"
struct Pair {{ int x, y; }};
extern "C" unsigned children(int directed, int decision, int a, int b, const int* l, const int* r, int* next, int64_t at,
                             int64_t cap) {{
  if (directed) walk_children<true>(decision, a, b, l, r, reinterpret_cast<Pair*>(next), at, cap);
  else walk_children<false>(decision, a, b, l, r, reinterpret_cast<Pair*>(next), at, cap);
  return directed ? walk_child_count<true>(decision) : walk_child_count<false>(decision);
}}
''')
    subprocess.run([build._cxx(), "-std=c++17", "-O1", "-shared", "-fPIC", "-o", str(d / "shim.so"),
                    str(d / "shim.cpp")], check=True)
    f = ctypes.CDLL(str(d / "shim.so")).children
    f.argtypes = [ctypes.c_int] * 4 + [ctypes.c_void_p] * 3 + [ctypes.c_int64] * 2
    f.restype = ctypes.c_uint
    return f


def _expected(directed, decision, a, b):
    if decision == SELF:
        kids = [(LEFT[a], LEFT[a]), (RIGHT[a], RIGHT[a]), (LEFT[a], RIGHT[a])]
        return kids + ([(RIGHT[a], LEFT[a])] if directed else [])
    if decision == SPLIT_A:
        return [(LEFT[a], b), (RIGHT[a], b)]
    if decision == SPLIT_B:
        return [(a, LEFT[b]), (a, RIGHT[b])]
    return []


@pytest.mark.parametrize("directed", [0, 1])
@pytest.mark.parametrize("decision,a,b", [(SELF, 1, 1), (SPLIT_A, 1, 2), (SPLIT_B, 1, 2), (FAR, 1, 2), (NEAR, 3, 4),
                                          (NONE, 3, 3)])
def test_every_place_below_the_end_is_written(fn, directed, decision, a, b):
    want = _expected(directed, decision, a, b)
    at = 5
    for cap in range(at - 2, at + 7):
        buf = np.full((16, 2), -1, np.int32)
        count = fn(directed, decision, a, b, LEFT.ctypes.data, RIGHT.ctypes.data, buf.ctypes.data, at, cap)
        assert count == len(want)
        full = np.full((16, 2), -1, np.int32)
        for k, pair in enumerate(want):
            if at + k < cap:
                full[at + k] = pair
        assert np.array_equal(buf, full), cap
