"""lbgb_batch_plan on the CPU: the tasks of a launch cover every instance once,
planning takes time in proportion to the instances and tasks however wide an
instance is, and what would be too many tasks is refused without being built."""

import ctypes
import time

import numpy as np
import pytest

from latticeboltzmann_gb300 import _lib
from test_abi_host import lib  # noqa: F401

P, C, L = _lib.PERIODIC, _lib.CAVITY, _lib.BOUNDARY_CODES["cavity-ladd"]


def plan(lib, sizes, boundary, dtype, steps=0, capacity=None):
    nx = np.array([s[0] for s in sizes], np.int32)
    ny = np.array([s[1] for s in sizes], np.int32)
    kind, most, count = ctypes.c_int(-1), ctypes.c_int(-1), ctypes.c_longlong(-1)

    def call(tasks):
        rc = lib.lbgb_batch_plan(nx.ctypes.data, ny.ctypes.data, len(sizes), boundary, dtype, steps,
                                 ctypes.byref(kind), ctypes.byref(most), tasks.ctypes.data if len(tasks) else None,
                                 len(tasks), ctypes.byref(count))
        return rc
    tasks = np.zeros((capacity or 0, 4), np.int32)
    rc = call(tasks)
    if rc == _lib.OK and capacity is None and count.value:
        tasks = np.zeros((count.value, 4), np.int32)
        rc = call(tasks)
    return rc, kind.value, most.value, count.value, tasks


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
def test_tasks_cover_every_cell_once(lib, boundary, sizes, dtype, steps):  # noqa: F811
    rc, kind, most, count, tasks = plan(lib, sizes, boundary, dtype, steps)
    assert rc == _lib.OK and most > 1 and count == len(tasks)
    assert all((g == 1).all() for g in covered(sizes, kind, tasks))
    # fewer asked for: the first ones, and the same count
    some = plan(lib, sizes, boundary, dtype, steps, capacity=5)
    assert some[3] == count and np.array_equal(some[4], tasks[:5])


def test_very_wide_instance_is_planned_quickly(lib):  # noqa: F811
    t0 = time.perf_counter()
    rc, kind, _, count, tasks = plan(lib, [(8, 20_000_000)], P, _lib.F32)
    assert time.perf_counter() - t0 < 5.0
    assert rc == _lib.OK and kind == _lib.BATCH_MARCH and count >= 20_000_000 // 120
    assert tasks[:, 2].max() < 20_000_000 and (tasks[:, 3] >> 16 == 32).mean() > 0.99


def test_too_many_tasks_are_refused_without_building_them(lib):  # noqa: F811
    t0 = time.perf_counter()
    rc = plan(lib, [(2 ** 31 - 1, 2 ** 31 - 1)], P, _lib.F32)[0]
    assert rc == _lib.EINVAL and "too many tasks" in _lib.last_error()
    assert time.perf_counter() - t0 < 5.0
