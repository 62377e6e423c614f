"""The buffers that the dense drivers keep between calls are given back: the
list they wait in (csrc/alloc.h) is bounded and shared fairly by the devices,
and an allocation of the solver that finds no memory frees them and is tried
again.
"""
import ctypes as C
import os
import subprocess

import pytest

from mr3smp_b200 import build
from test_alloc_failure_cpu import _context, _solve, lib  # noqa: F401  (fixture)

HARNESS = r"""
#include "alloc.h"
struct Obj { int device, id; };
static KeptList<Obj, 4> g;
static Obj g_obj[64];
// give object id of a device: the id of the object to free, -1 for none
extern "C" int give(int device, int id) {
  g_obj[id] = {device, id};
  Obj *out = g.give(&g_obj[id]);
  return out ? out->id : -1;
}
extern "C" int take(int device) { Obj *x = g.take(device); return x ? x->id : -1; }
extern "C" int take_any() { Obj *x = g.take_any(); return x ? x->id : -1; }
"""


@pytest.fixture
def kept(tmp_path):
    (tmp_path / "h.cpp").write_text(HARNESS)
    so = str(tmp_path / "h.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I" + build.CSRC,
                    "-I/usr/local/cuda/include", "-o", so, str(tmp_path / "h.cpp")], check=True)
    return C.CDLL(so)


def test_bounded_and_taken_by_device(kept):
    assert [kept.give(0, k) for k in range(4)] == [-1] * 4
    assert kept.give(0, 4) == 4                 # full: the new one is freed
    assert kept.take(1) == -1
    assert sorted(kept.take(0) for _ in range(4)) == [0, 1, 2, 3]
    assert kept.take(0) == -1 and kept.take_any() == -1


def test_one_device_does_not_keep_the_places_from_another(kept):
    for k in range(4):
        kept.give(0, k)
    assert kept.give(1, 10) in (0, 1, 2, 3)     # device 1 gets a place
    assert kept.give(1, 11) in (0, 1, 2, 3)     # two each
    assert kept.give(1, 12) == 12
    assert kept.give(2, 20) in (0, 1, 2, 3, 10, 11)
    assert kept.take(2) == 20
    left = [kept.take_any() for _ in range(4)]
    assert left.count(-1) == 1 and len(set(left)) == 4


@pytest.mark.parametrize("idle", [1, 4])
def test_allocation_without_memory_frees_the_idle_buffers(lib, idle):  # noqa: F811
    retried = host = 0
    for k in range(1000):
        ctx = _context(lib)
        lib.fake_idle(idle)
        rc, _ = _solve(lib, ctx, 30, 2, 1000, 60, fail=k)
        tried = lib.fake_allocs()
        lib.mr3_cuda_ctx_destroy(ctx)
        freed = idle - lib.mr3_dense_release()
        if tried <= k:                          # the solve makes fewer allocations
            break
        assert (rc, freed) in ((0, idle), (2, 0)), k
        retried += rc == 0
        host += rc == 2                         # page-locked host buffers
    assert retried > 45 and host <= 4
