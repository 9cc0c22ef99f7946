"""The order of launches of a run (csrc/lbgb_run.h), compiled for the host: the
stochastic-rounding counter moves by the steps that were launched, also where a
launch in the middle of the run fails."""

import ctypes
import os
import subprocess

import pytest

from latticeboltzmann_gb300 import _build

SOURCE = r"""
#include "lbgb_run.h"
extern "C" int run(int nsteps, int most, int fail_at, int bump_rc, int *launched, int *offsets, int *counter) {
    *launched = 0;
    return lbgb::run_counted_steps(
        nsteps, [&](int left) { return left < most ? left : most; },
        [&](int n, int done) {
            if (*launched == fail_at) return 7;
            offsets[(*launched)++] = done;
            return 0;
        },
        [&](int n) {
            *counter += n;
            return bump_rc;
        });
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("run")
    (d / "run.cpp").write_text(SOURCE)
    so = str(d / "run.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", _build.CSRC, "-o", so, str(d / "run.cpp")],
                   check=True)
    lib = ctypes.CDLL(so)

    def call(nsteps, most, fail_at=-1, bump_rc=0):
        launched, counter, offsets = ctypes.c_int(0), ctypes.c_int(0), (ctypes.c_int * 64)()
        rc = lib.run(nsteps, most, fail_at, bump_rc, ctypes.byref(launched), offsets, ctypes.byref(counter))
        return rc, list(offsets[:launched.value]), counter.value
    return call


@pytest.mark.parametrize("nsteps,most", [(0, 4), (1, 4), (4, 4), (11, 4), (10, 6), (7, 1)])
def test_whole_runs(run, nsteps, most):
    assert run(nsteps, most) == (0, list(range(0, nsteps, most)), nsteps)


@pytest.mark.parametrize("fail_at", [0, 1, 2])
def test_a_launch_that_fails(run, fail_at):
    assert run(11, 4, fail_at) == (7, list(range(0, 4 * fail_at, 4)), 4 * fail_at)
    assert run(11, 4, fail_at, 9)[0] == 7


def test_a_counter_that_fails(run):
    assert run(11, 4, bump_rc=9) == (9, [0, 4, 8], 11)
