"""wide_tree (nuray_gb300/csrc/host_scene.cpp): the device walks the four-wide
tree on a stack without a full test, so no ray may need more entries than the
array has, a ray that passes every slot's test included (a direction of NaN
passes the empty boxes of unused slots too). On the CPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from nuray_gb300.build import _cuda_home

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "nuray_gb300", "csrc")
OUT = os.path.join(ROOT, "tests", "_build")
LIMIT = 96  # NR_STACK_LIMIT

SHIM = """
#include <cstring>
#include "host_scene.h"
#include "nr_types.h"
extern "C" int stack_limit() { return NR_STACK_LIMIT; }
extern "C" int tree(const int* refs, const float* box, int n, int limit, int* kids) {
    const auto w = nr::wide_tree(refs, box, n, 1e-3f, limit);
    for (size_t i = 0; i < w.size(); ++i) std::memcpy(kids + 4 * i, w[i].ref, 16);
    return (int)w.size();
}
extern "C" int need(const int* refs, const float* box, int n, int width) {
    std::vector<nr::WideNodeHost> w;
    return nr::build_wide(refs, box, n, 1e-3f, width, w);
}
"""


@pytest.fixture(scope="module")
def tree_lib():
    os.makedirs(OUT, exist_ok=True)
    src, lib = os.path.join(OUT, "stack_shim.cpp"), os.path.join(OUT, "libstack_shim.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-ffp-contract=off", "-shared", "-I", CSRC, "-I",
                    os.path.join(ROOT, "include"), "-I", os.path.join(_cuda_home(), "include"), src,
                    os.path.join(CSRC, "host_scene.cpp"), os.path.join(CSRC, "image_io.cpp"),
                    os.path.join(CSRC, "jpeg.cpp"), "-o", lib, "-lpthread"], check=True)
    return ctypes.CDLL(lib)


def _chain(length, cluster, rng):
    """A binary tree in depth-first order: a chain of `length` inner nodes,
    each with the next of them and a cluster (a full subtree of `cluster`
    leaves, or a leaf) for children; boxes of random sizes."""
    refs, boxes = [], []

    def box(scale):
        lo = rng.uniform(-10, 10, 3)
        return np.concatenate([lo, lo + rng.uniform(0.1, scale, 3)])

    def sub(leaves):
        if leaves == 1:
            return -2
        me = len(refs)
        refs.append(None), boxes.append(np.concatenate([box(2), box(2)]))
        refs[me] = (sub(leaves // 2), sub(leaves - leaves // 2))
        return me

    def link(k):
        if k == 0:
            return sub(cluster)
        me = len(refs)
        refs.append(None), boxes.append(np.concatenate([box(30), box(30)]))
        refs[me] = (sub(cluster), link(k - 1))
        return me

    link(length)
    return np.array(refs, np.int32).reshape(-1, 2), np.array(boxes, np.float32).reshape(-1, 12)


def _deepest(kids):
    """Entries of a walk that enters every slot: three pushed at every node, the
    deepest child taken last. Children follow their parent."""
    need = np.zeros(len(kids), np.int64)
    for i in range(len(kids) - 1, -1, -1):
        inner = kids[i][kids[i] >= 0]
        need[i] = 3 + (need[inner].max() if len(inner) else 0)
    return int(need[0])


@pytest.mark.parametrize("cluster", [1, 2, 3, 4, 8, 9])
@pytest.mark.parametrize("length", [1, 2, 10, 29, 30, 31, 32, 33, 45, 60, 80, 90])
def test_every_ray_stays_on_the_stack(tree_lib, length, cluster):
    assert tree_lib.stack_limit() == LIMIT
    refs, box = _chain(length, cluster, np.random.default_rng(100 * length + cluster))
    p = [a.ctypes.data_as(ctypes.c_void_p) for a in (refs, box)]
    need = tree_lib.need(*p, len(refs), 4)
    kids = np.zeros((len(refs), 4), np.int32)
    for limit in (LIMIT, need + 1, need + 2, need + 3):
        n = tree_lib.tree(*p, len(refs), limit, kids.ctypes.data_as(ctypes.c_void_p))
        assert (n > 0) == (need + 2 <= limit)  # the whole of the range that fits keeps its tree
        if n:
            assert _deepest(kids[:n]) <= limit


def test_trees_without_inner_nodes(tree_lib):
    assert tree_lib.tree(None, None, 0, LIMIT, None) == 0
