"""overlap.h, compiled for the host, against sets of bytes."""
import ctypes as C
import os
import random
import subprocess

import pytest

from tests.conftest import ROOT

SOURCE = """
#include "overlap.h"
extern "C" int meet(const long long* a, const long long* b) {
  auto rows = [](const long long* v) { return adk::ByteRows{(intptr_t)v[0], (uint32_t)v[1], (uint32_t)v[2], v[3], v[4], v[5], v[6]}; };
  return adk::rows_meet(rows(a), rows(b));
}
"""


@pytest.fixture(scope="module")
def meet(tmp_path_factory):
    d = tmp_path_factory.mktemp("overlap")
    (d / "o.cc").write_text(SOURCE)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(ROOT, "arraydiff_cuda_b200", "csrc"), str(d / "o.cc"), "-o", str(d / "o.so")])
    L = C.CDLL(str(d / "o.so"))
    return lambda a, b: bool(L.meet((C.c_longlong * 7)(*a), (C.c_longlong * 7)(*b)))


def _bytes(base, N, H, sn, sy, lo, hi):
    return {base + n * sn + y * sy + i for n in range(N) for y in range(H) for i in range(lo, hi)}


def test_against_sets(meet):
    rng = random.Random(11)
    seen = [0, 0]
    for _ in range(6000):
        def rows(base):
            lo = -rng.randint(0, 4)
            return (base, rng.randint(0, 3), rng.randint(0, 4), rng.choice([-1, 1]) * rng.randint(0, 60), rng.choice([-1, 1, 1]) * rng.randint(0, 20), lo,
                    lo + rng.randint(1, 9))
        a, b = rows(1000), rows(1000 + rng.randint(-60, 60))
        want = bool(_bytes(*a) & _bytes(*b))
        seen[want] += 1
        assert meet(a, b) == want and meet(b, a) == want
    assert min(seen) > 1000


def test_views_of_one_buffer(meet):
    y = (4096, 2, 5, 5 * 64, 64, 0, 32)                       # the left half of every row
    assert not meet(y, (4096 + 32, 2, 5, 5 * 64, 64, 0, 32))  # the right half
    assert not meet(y, (4096 + 2 * 5 * 64, 2, 5, 5 * 64, 64, 0, 32))
    assert meet(y, y) and meet(y, (4096 + 30, 2, 5, 5 * 64, 64, 0, 32)) and meet(y, (4096 + 64, 2, 5, 5 * 64, 64, 0, 32))
    even, odd = (0, 3, 4, 2 * 4 * 32, 32, 0, 32), (4 * 32, 3, 4, 2 * 4 * 32, 32, 0, 32)
    assert not meet(even, odd)                                # every other image
