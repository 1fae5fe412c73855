"""Choices of the fp32 convolutions that need no GPU: conv_f32_plan.h, compiled for the host."""
import ctypes as C
import os
import random
import subprocess

import pytest

from tests.conftest import ROOT

SOURCE = """
#include "conv_f32_plan.h"
extern "C" uint32_t cluster_size(const uint32_t* held, unsigned long long tiles, uint32_t steps, uint32_t most) {
  return adk::f32_cluster_size([=](uint32_t cs) { return held[__builtin_ctz(cs)]; }, tiles, steps, most, 148);
}
extern "C" uint32_t largest_cluster(const uint32_t* held, uint32_t most) {
  return adk::f32_largest_cluster([=](uint32_t cs) { return held[__builtin_ctz(cs)]; }, most);
}
extern "C" uint32_t k3_split(unsigned long long tiles, unsigned long long all, unsigned long long words, uint32_t per_sm) {
  const adk::F32Split s = adk::f32_k3_split(tiles, all, words, 148, per_sm);
  return s.cs << 16 | s.slices;
}
extern "C" uint32_t few_images(uint32_t N, unsigned long long image, unsigned long long z, unsigned long long limit) {
  return adk::f32_few_images(N, image, z, limit);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cc").write_text(SOURCE)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(ROOT, "arraydiff_cuda_b200", "csrc"),
                           "-I", os.path.join(ROOT, "include"), str(d / "plan.cc"), "-o", str(d / "plan.so")])
    L = C.CDLL(str(d / "plan.so"))
    L.cluster_size.argtypes = [C.POINTER(C.c_uint32), C.c_uint64, C.c_uint32, C.c_uint32]
    L.largest_cluster.argtypes = [C.POINTER(C.c_uint32), C.c_uint32]
    L.k3_split.argtypes = [C.c_uint64, C.c_uint64, C.c_uint64, C.c_uint32]
    L.few_images.argtypes = [C.c_uint32, C.c_uint64, C.c_uint64, C.c_uint64]
    L.k3_split.restype = L.cluster_size.restype = L.largest_cluster.restype = L.few_images.restype = C.c_uint32
    return L


FULL = [296, 148, 74, 33, 14]      # clusters of 1, 2, 4, 8, 16 CTAs on a whole GPU, two CTAs per SM


def _held(missing):
    return [0 if i in missing else n for i, n in enumerate(FULL)]


@pytest.mark.parametrize("missing", [(), (4,), (3, 4), (2, 3, 4), (1, 2, 3, 4), (3,), (1, 3)])
def test_a_cluster_that_the_device_does_not_hold_is_not_chosen(plan, missing):
    held = _held(missing)
    h = (C.c_uint32 * 5)(*held)
    rng = random.Random(5)
    seen = set()
    for _ in range(2000):
        tiles, steps, most = int(2 ** rng.uniform(0, 12)), int(2 ** rng.uniform(0, 10)), rng.choice([1, 8, 16])
        cs = plan.cluster_size(h, tiles, steps, most)
        assert held[cs.bit_length() - 1] and cs <= most and (cs == 1 or steps >= 4 * cs)
        seen.add(cs)
    assert seen == {1 << i for i in range(5) if held[i]}
    for most in (1, 2, 4, 8, 16):
        cs = plan.largest_cluster(h, most)
        assert held[cs.bit_length() - 1] and cs == max(1 << i for i in range(5) if held[i] and 1 << i <= most)


def test_clusters_of_16(plan):
    """The layers of tests/test_gpu_conv_f32.py that are there for them: tiles and stages of each pass."""
    for held in (FULL, [444, 222, 111, 50, 21]):       # two or three CTAs per SM
        h = (C.c_uint32 * 5)(*held)
        for tiles, steps in ((3, 128 * 9 // 16), (2, 130 * 9 // 16), (1, 120 * 9 // 16)):
            assert plan.cluster_size(h, tiles, steps, 16) == 16


def test_nothing_known_about_the_device(plan):
    h = (C.c_uint32 * 5)()
    assert plan.cluster_size(h, 16, 1024, 16) == 1 and plan.largest_cluster(h, 8) == 1


@pytest.mark.parametrize("N,image,z,limit", [
    (90, 3 * 4000 * 4000, 64 * 64 * 3 * 4 * 4, 64 << 20),   # the gradient has more than 2^32 elements, dy 65 thousand
    (89, 3 * 4000 * 4000, 64 * 64 * 3 * 4 * 4, 64 << 20),   # just below: the step of the grid would pass 2^32
    (5, 2 ** 31 - 1, 1 << 20, 64 << 20), (3, 2 ** 30, 1 << 20, 64 << 20),
    (5, 8 * 134 * 134, 25690112, 64 << 20),                 # the scratch is the limit: pieces of 2, 2, 1
    (4, 3 * 224 * 224, 3 * 49 * 218 * 218 * 4, 64 << 20), (1, 1, 4, 64 << 20),
    (2, 100, (64 << 20) + 4, 64 << 20),                     # one image is too large: not this way
])
def test_pieces_of_the_gradient_into_few_channels(plan, N, image, z, limit):
    """32-bit indices hold the elements of a piece and a step of the grid (148 x 16 blocks of 256) more."""
    n = plan.few_images(N, image, z, limit)
    most = max(i for i in range(N + 1) if i * z <= limit and i * image < 2 ** 31)
    assert n == most and n * image + 148 * 16 * 256 < 2 ** 32


def test_filter_gradient_split_depends_on_its_arguments_alone(plan):
    """The same split whatever was asked for before; at least two stages per CTA, at most 16 slices and 32 MB of them."""
    rng = random.Random(6)
    calls = []
    for _ in range(500):
        tiles, stages, words = int(2 ** rng.uniform(0, 9)), int(2 ** rng.uniform(0, 12)), int(2 ** rng.uniform(10, 23))
        calls.append((tiles, stages, words, rng.choice([2, 3])))
    first = [plan.k3_split(*c) for c in calls]
    assert [plan.k3_split(*c) for c in reversed(calls)] == first[::-1]
    assert any(plan.k3_split(t, s, w, 2) != plan.k3_split(t, s, w, 3) for t, s, w, _ in calls)
    for (tiles, stages, words, _), split in zip(calls, first):
        cs, slices = split >> 16, split & 0xffff
        assert cs in (1, 2, 4, 8) and 1 <= slices <= 16
        assert cs * slices == 1 or stages >= 2 * cs * slices
        assert slices == 1 or slices * words * 4 <= 32 << 20
