"""lbgb_batch_plan on the CPU: the tasks of a launch cover every instance once,
planning takes time in proportion to the instances and tasks however wide an
instance is, what would be too many tasks is refused without being built, and
batches whose several steps per launch measured slower than one take one.  The
last is asked of the planner itself (csrc/lbgb_batch_plan.h), compiled for the
host, for a GPU of 152 SMs."""

import ctypes
import os
import subprocess
import time

import numpy as np
import pytest

from latticeboltzmann_gb300 import _build, _lib
from test_abi_host import lib  # noqa: F401

P, C, L = _lib.PERIODIC, _lib.CAVITY, _lib.BOUNDARY_CODES["cavity-ladd"]


ELEMENT = {_lib.F32: 4, _lib.F64: 8, _lib.F16DEV: 2, _lib.BF16DEV: 2, _lib.F32DEV: 4}
SOURCE = r"""
#include "lbgb_batch_plan.h"
extern "C" int form(const int *nx, const int *ny, int n, int boundary, int dtype, int element, int steps, int *most,
                    int *tasks, long long capacity, long long *count) {
    const lbgb::BatchForm f = lbgb::batch_form(nx, ny, n, boundary, dtype, element, steps, 152,
                                               lbgb::BatchSink{reinterpret_cast<lbgb::BatchTask *>(tasks), capacity});
    *most = f.most;
    *count = f.n_tasks;
    return f.kind;
}
// cycles of a step: tiles, one step per launch
extern "C" void lattice_costs(int nx, int ny, int element, double *c) {
    lbgb::TilePlan p;
    lbgb::tile_plan(p, nx, ny, 0, element, 1.45, 152);
    c[0] = p.cost;
    c[1] = lbgb::single_cost((double)nx * ny, element, 152);
}
"""


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE)
    so = str(d / "plan.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc()))), "include")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", _build.INCLUDE, "-I", _build.CSRC, "-I", cuda,
                    "-o", so, str(d / "plan.cpp")], check=True)
    return ctypes.CDLL(so)


def form(planner, sizes, boundary, dtype, steps=0, capacity=0):
    """(kind, most, count, the first ``capacity`` tasks) on 152 SMs."""
    nx, ny = (np.array([s[i] for s in sizes], np.int32) for i in (0, 1))
    most, count, tasks = ctypes.c_int(-1), ctypes.c_longlong(-1), np.zeros((capacity, 4), np.int32)
    ptr = lambda a: ctypes.c_void_p(a.ctypes.data)
    kind = planner.form(ptr(nx), ptr(ny), len(sizes), boundary, dtype, ELEMENT[dtype], steps, ctypes.byref(most),
                        ptr(tasks), ctypes.c_longlong(capacity), ctypes.byref(count))
    return kind, most.value, count.value, tasks


def plan(lib, sizes, boundary, dtype):
    """lbgb_batch_plan, asked for the count only."""
    nx, ny = (np.array([s[i] for s in sizes], np.int32) for i in (0, 1))
    kind, most, count = ctypes.c_int(-1), ctypes.c_int(-1), ctypes.c_longlong(-1)
    rc = lib.lbgb_batch_plan(nx.ctypes.data, ny.ctypes.data, len(sizes), boundary, dtype, 0, ctypes.byref(kind),
                             ctypes.byref(most), None, 0, ctypes.byref(count))
    return rc, kind.value, most.value, count.value


def covered(sizes, kind, tasks):
    """How often each cell of each instance is written."""
    grids = [np.zeros(s, np.int32) for s in sizes]
    for b, x, y, w in tasks.tolist():
        nx, ny = sizes[b]
        if kind == _lib.BATCH_TILE:
            grids[b][x:x + (w & 0xffff), y:y + (w >> 16)] += 1
        else:
            rows, lanes = w & 0xffff, w >> 16
            assert rows + 4 <= nx
            grids[b][x:x + rows * (32 // lanes), y:y + 4 * (lanes - 2)] += 1
    return grids


UNEVEN = [(8, 16), (9, 17), (40, 25), (33, 56), (21, 120), (70, 121), (130, 145), (8, 5000), (1100, 511), (1024, 512)]


@pytest.mark.parametrize("boundary", [P, C, L])
@pytest.mark.parametrize("sizes,dtype,steps", [(UNEVEN, _lib.F32, 4), (UNEVEN, _lib.F32, 2), (UNEVEN[:7], _lib.F64, 0),
                                               ([(5, 3), (2, 2), (64, 33), (9, 300), (300, 9)], _lib.F32DEV, 3)])
def test_tasks_cover_every_cell_once(planner, boundary, sizes, dtype, steps):
    kind, most, count, _ = form(planner, sizes, boundary, dtype, steps)
    assert kind != _lib.BATCH_SINGLE and most > 1 and count > 5
    tasks = form(planner, sizes, boundary, dtype, steps, count)[3]
    assert all((g == 1).all() for g in covered(sizes, kind, tasks))
    # fewer asked for: the first ones, and the same count
    some = form(planner, sizes, boundary, dtype, steps, 5)
    assert some[2] == count and np.array_equal(some[3], tasks[:5])


def test_very_wide_instance_is_planned_quickly(lib, planner):  # noqa: F811
    t0 = time.perf_counter()
    rc, kind, _, count = plan(lib, [(8, 20_000_000)], P, _lib.F32)
    tasks = form(planner, [(8, 20_000_000)], P, _lib.F32, 0, 1_000_000)[3]
    assert time.perf_counter() - t0 < 5.0
    assert rc == _lib.OK and kind == _lib.BATCH_MARCH and 20_000_000 // 120 <= count < 1_000_000
    assert (tasks[:count, 3] >> 16 == 32).mean() > 0.99 and tasks[:count, 2].max() < 20_000_000


def test_too_many_tasks_are_refused_without_building_them(lib):  # noqa: F811
    t0 = time.perf_counter()
    rc = plan(lib, [(2 ** 31 - 1, 2 ** 31 - 1)], P, _lib.F32)[0]
    assert rc == _lib.EINVAL and "too many tasks" in _lib.last_error()
    assert time.perf_counter() - t0 < 5.0


@pytest.mark.parametrize("sizes,boundary,dtype,kind", [
    # several steps per launch measured 4, 2 and 11 times as slow as one
    ([(16, 16)] * 8000, C, _lib.F32, _lib.BATCH_SINGLE),
    ([(32, 32)] * 3000, C, _lib.F32, _lib.BATCH_SINGLE),
    ([(4, 4)] * 68750, P, _lib.F32, _lib.BATCH_SINGLE),
    ([(4, 4)] * 8750, C, _lib.F64, _lib.BATCH_SINGLE),
    ([(8, 8)] * 17187, L, _lib.F16DEV, _lib.BATCH_SINGLE),
    # and faster
    ([(400, 400)] * 62, C, _lib.F32, _lib.BATCH_MARCH),
    ([(256, 256)] * 152, L, _lib.F32DEV, _lib.BATCH_MARCH),
    ([(300, 333), (120, 240), (64, 800)] * 10, P, _lib.F32, _lib.BATCH_MARCH),
    ([(256, 256)], L, _lib.F32DEV, _lib.BATCH_TILE),
    ([(64, 64)] * 200, C, _lib.F32, _lib.BATCH_TILE),
    ([(64, 64)] * 10, P, _lib.F64, _lib.BATCH_TILE),
])
def test_form_of_a_batch(planner, sizes, boundary, dtype, kind):
    """It does not depend on the steps asked for."""
    for steps in (0, 1, 2, 4):
        got, most, count, _ = form(planner, sizes, boundary, dtype, steps)
        assert got == kind
        assert (most, count) == (1, 0) if kind == _lib.BATCH_SINGLE else (most > 1 and count > 0)


@pytest.mark.parametrize("size,element,tiles", [((2, 400_000), 4, False), ((2, 400_000), 2, False),
                                                ((5, 200_000), 2, False), ((256, 256), 4, True), ((256, 256), 2, True),
                                                ((960, 976), 4, True), ((1000, 1096), 2, True), ((16, 56_000), 4, True)])
def test_lattices_a_few_rows_high_take_one_step_per_launch(planner, size, element, tiles):
    c = np.zeros(2)
    planner.lattice_costs(*size, element, ctypes.c_void_p(c.ctypes.data))
    assert (c[0] < c[1]) == tiles
