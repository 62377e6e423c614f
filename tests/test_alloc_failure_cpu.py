"""A device allocation that fails leaves the solver's context usable: the call
returns its error, and the next call, which needs less, allocates what it
needs and passes no null buffer to a kernel.  The solver's host code runs on
a CUDA runtime of the test's own (tests/fake_cudart.cpp) in which every
allocation of a solve is made to fail in turn.
"""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

from mr3smp_b200 import CudaProb, build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _pointer_parameters():
    """Kernel name -> positions of its pointer parameters, from the source."""
    src = open(os.path.join(build.CSRC, "solver.cu")).read()
    src = re.sub(r"//[^\n]*", "", src)
    out = {}
    for m in re.finditer(r"__global__ void[^;{]*?\b(k_\w+)\(([^;{]*?)\)\s*\{", src):
        args = m.group(2).split(",")
        out[m.group(1)] = [i for i, a in enumerate(args) if "*" in a]
    return out


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    obj = os.path.join(build.BUILD, "solver.cu.o")
    if not build.up_to_date() or not os.path.exists(obj):
        build.build(force=True)
    so = str(tmp_path_factory.mktemp("fake") / "solver_fake.so")
    # (-Bsymbolic: its own runtime, whatever libraries the process has loaded)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic",
                    "-I/usr/local/cuda/include", "-o", so,
                    os.path.join(ROOT, "tests", "fake_cudart.cpp"), obj], check=True)
    L = C.CDLL(so)
    L.fake_launches.restype = C.c_char_p
    L.fake_allocs.restype = C.c_long
    L.fake_fail.argtypes = [C.c_long]
    L.mr3_cuda_solve.argtypes = [C.c_void_p, C.c_int, C.POINTER(CudaProb), C.c_void_p]
    L.mr3_cuda_ctx_destroy.argtypes = [C.c_void_p]
    L.mr3_cuda_ws.argtypes = [C.c_void_p, C.c_int, C.c_size_t]
    L.mr3_cuda_ws.restype = C.c_void_p
    pointers = _pointer_parameters()
    assert len(pointers) > 40
    for name, at in pointers.items():
        L.fake_ptr_args(name.encode(), (C.c_int * len(at))(*at), len(at))
    return L


def _context(L):
    ctx = C.c_void_p()
    L.fake_fail(-1)
    assert L.mr3_cuda_ctx_create(0, C.byref(ctx)) == 0
    return ctx


def _solve(L, ctx, n, count, arena, nsng, fail=-1):
    """One solve of `count` problems; two levels of a cluster, their arena and
    nsng singletons.  (return code, launches with their null pointers)"""
    keep = [np.zeros(n * (n + 5)) for _ in range(count)]
    probs = (CudaProb * count)()
    for p, a in zip(probs, keep):
        at = a.ctypes.data
        p.n, p.jobz, p.range, p.ldz = n, 1, 1, n
        p.D, p.E, p.W, p.Zsupp, p.Z = at, at + 8 * n, at + 16 * n, at + 24 * n, at + 40 * n
    lv = [1, 0, 0, 1, arena, nsng, 0, 0, nsng]
    L.fake_levels((C.c_int * len(lv))(*lv), len(lv))
    L.fake_clear()
    L.fake_fail(fail)
    rc = L.mr3_cuda_solve(ctx, count, probs, None)
    return rc, L.fake_launches().decode()


@pytest.mark.parametrize("finish_max", ["0", "1000000"])   # with and without the rounds' scratch
def test_next_solve_after_a_failed_allocation(lib, finish_max, monkeypatch):
    monkeypatch.setenv("MR3_FINISH_MAX", finish_max)
    small, big = (30, 2, 1000, 60), (60, 3, 5000, 180)
    ctx = _context(lib)
    rc, want = _solve(lib, ctx, *small)
    assert rc == 0 and "k_sng_finish" in want and "k_cl_rrf" in want
    lib.mr3_cuda_ctx_destroy(ctx)
    ctx = _context(lib)
    rc, _ = _solve(lib, ctx, *big)
    total = lib.fake_allocs()
    assert rc == 0 and total > 50
    lib.mr3_cuda_ctx_destroy(ctx)
    for first in (None, small):      # a new context, one that has solved before
        for k in range(total):
            ctx = _context(lib)
            if first:
                assert _solve(lib, ctx, *first)[0] == 0
            rc, _ = _solve(lib, ctx, *big, fail=k)
            failed = lib.fake_allocs() > k
            assert rc == (2 if failed else 0), k
            rc, got = _solve(lib, ctx, *small)
            assert rc == 0, (first, k)
            assert got == want, (first, k)
            lib.mr3_cuda_ctx_destroy(ctx)


def test_failed_workspace(lib):
    """A workspace that could not be had does not make the next solve fail."""
    ctx = _context(lib)
    lib.fake_fail(0)
    assert not lib.mr3_cuda_ws(ctx, 0, 1 << 20)
    assert _solve(lib, ctx, 30, 2, 1000, 60)[0] == 0
    assert lib.mr3_cuda_ws(ctx, 0, 1 << 10)
    lib.mr3_cuda_ctx_destroy(ctx)
