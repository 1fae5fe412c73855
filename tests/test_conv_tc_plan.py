"""Choices of the tensor-core convolutions that need no GPU: conv_tc_plan.h, compiled for the host."""
import ctypes as C
import os
import random
import subprocess

import pytest

from tests.conftest import ROOT

SOURCE = """
#include "conv_tc_plan.h"
extern "C" uint32_t wgrad_splits(uint32_t sp, uint32_t K, uint32_t C, uint32_t taps) { return adk::tc::wgrad_splits(sp, K, C, taps, 148); }
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cc").write_text(SOURCE)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(ROOT, "arraydiff_cuda_b200", "csrc"), str(d / "plan.cc"),
                           "-o", str(d / "plan.so")])
    L = C.CDLL(str(d / "plan.so"))
    L.wgrad_splits.argtypes = [C.c_uint32] * 4
    L.wgrad_splits.restype = C.c_uint32
    return L


def test_filter_gradient_splits_keep_the_runs_of_sums_short(plan):
    """An accumulator rounds towards zero at every step, so its error grows with the pixels that it sums: never fewer splits than make
    two items per SM, unless 64 are enough or there are no more tiles of pixels."""
    rng = random.Random(7)
    cases = [(512, 256, 1024, 1), (16, 512, 512, 9), (152, 256, 128, 9), (1, 64, 64, 9), (3000, 64, 64, 1), (7, 2048, 512, 1)]
    cases += [(int(2 ** rng.uniform(0, 14)), rng.choice([32, 64, 128, 256, 512, 1024, 2048]), 64 * int(2 ** rng.uniform(0, 5)), rng.choice([1, 4, 9, 25]))
              for _ in range(3000)]
    more = 0
    for sp, K, Cc, taps in cases:
        n = plan.wgrad_splits(sp, K, Cc, taps)
        bn = 128 if Cc > 64 else 64
        items = taps * -(-K // 128) * -(-Cc // bn)
        least = min(-(-2 * 148 // items), sp, 64)
        assert least <= n <= min(sp, 64)
        more += n > least
    assert more > 100
