"""build_wide (nuray_gb300/csrc/host_scene.cpp): the four-wide tree of the
device's walks for few rays, on the CPU. It has to hold every leaf of the
binary tree once, in order, under boxes that are the binary tree's widened by
the given amount, with children after their parent, and to say how deep a
stack its walk needs."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "nuray_gb300", "csrc")
OUT = os.path.join(ROOT, "tests", "_build")

SHIM = """
#include <cstring>
#include "host_scene.h"
extern "C" int wide(const int* refs, const float* box, int n, float delta, int width, float* planes, int* kids, int* nodes) {
    std::vector<nr::WideNodeHost> w;
    const int need = nr::build_wide(refs, box, n, delta, width, w);
    for (size_t i = 0; i < w.size(); ++i) {
        std::memcpy(planes + 24 * i, w[i].plane, 96);
        std::memcpy(kids + 4 * i, w[i].ref, 16);
    }
    *nodes = (int)w.size();
    return need;
}
"""


@pytest.fixture(scope="module")
def wide_lib():
    os.makedirs(OUT, exist_ok=True)
    src, lib = os.path.join(OUT, "wide_shim.cpp"), os.path.join(OUT, "libwide_shim.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-ffp-contract=off", "-shared", "-I", CSRC, "-I",
                    os.path.join(ROOT, "include"), src, os.path.join(CSRC, "host_scene.cpp"),
                    os.path.join(CSRC, "image_io.cpp"), os.path.join(CSRC, "jpeg.cpp"), "-o", lib, "-lpthread"], check=True)
    return ctypes.CDLL(lib)


def _tree(leaves, shape, rng):
    """A binary tree over `leaves` leaf boxes: references (leaf k of k % 5 + 1
    triangles from 8 k on) and per inner node both children's boxes, inner
    nodes depth-first."""
    lo = rng.uniform(-10, 10, (leaves, 3)).astype(np.float32)
    hi = lo + rng.uniform(0, 2, (leaves, 3)).astype(np.float32)
    refs, boxes = [], []

    def build(a, b):
        if b - a == 1:
            return -1 - ((8 * a << 3) | (a % 5 + 1)), lo[a], hi[a]
        m = {"even": (a + b) // 2, "left": b - 1, "right": a + 1}.get(shape) or int(rng.integers(a + 1, b))
        me = len(refs)
        refs.append(None), boxes.append(None)
        l, r = build(a, m), build(m, b)
        refs[me] = (l[0], r[0])
        boxes[me] = np.concatenate([l[1], l[2], r[1], r[2]])
        return me, np.minimum(l[1], r[1]), np.maximum(l[2], r[2])

    build(0, leaves)
    return np.array(refs, np.int32).reshape(-1, 2), np.array(boxes, np.float32).reshape(-1, 12), lo, hi


@pytest.mark.parametrize("width", [2, 3, 4])
@pytest.mark.parametrize("shape", ["even", "left", "right", "any"])
@pytest.mark.parametrize("leaves", [2, 3, 4, 5, 8, 17, 64, 333])
def test_wide_tree(wide_lib, leaves, shape, width):
    rng = np.random.default_rng(leaves)
    refs, box, lo, hi = _tree(leaves, shape, rng)
    n, delta = len(refs), np.float32(1e-3)
    planes, kids = np.zeros((n, 6, 4), np.float32), np.zeros((n, 4), np.int32)
    count = ctypes.c_int()
    need = wide_lib.wide(refs.ctypes.data_as(ctypes.c_void_p), box.ctypes.data_as(ctypes.c_void_p), n,
                         ctypes.c_float(delta), width, planes.ctypes.data_as(ctypes.c_void_p),
                         kids.ctypes.data_as(ctypes.c_void_p), ctypes.byref(count))
    w = count.value
    assert 1 <= w <= n
    seen = []

    def visit(i):
        """Leaves below node i in order; checks boxes; returns the deepest stack a walk needs."""
        own, deep, inside_lo, inside_hi = 0, 0, [], []
        for k in range(4):
            p = planes[i, :, k]
            if np.all(p[0::2] == np.inf):  # unused: an empty box and an empty leaf
                assert np.all(p[1::2] == -np.inf) and kids[i, k] == -1
                continue
            own += 1
            if kids[i, k] < 0:
                a = (-1 - kids[i, k]) >> 6
                seen.append(a)
                assert (-1 - kids[i, k]) & 7 == a % 5 + 1
                np.testing.assert_array_equal(p[0::2], lo[a] - delta)
                np.testing.assert_array_equal(p[1::2], hi[a] + delta)
            else:
                assert i < kids[i, k] < w
                s, l, h = visit(kids[i, k])
                deep = max(deep, s)
                assert np.all(p[0::2] <= l) and np.all(p[1::2] >= h)  # a box holds its children's
            inside_lo.append(p[0::2]), inside_hi.append(p[1::2])
        assert 2 <= own <= width
        return own - 1 + deep, np.min(inside_lo, 0), np.max(inside_hi, 0)

    stack = visit(0)[0]
    assert seen == list(range(leaves)) and stack == need
