"""The fixed-point FP64 collision and fields (csrc/lbgb_fix64.cuh), compiled
for the host: against extended precision over random states, next to the FP64
evaluation they replace; the conversions over their whole range; and which
nodes are refused (they take the FP64 evaluation).

Tolerances: the largest error is below the FP64 evaluation's on the same
states; mass and momentum of a node move by less than the nine stored values'
roundings, half a last place of 1/2 each."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#define __host__
#define __device__
#define __forceinline__ inline
#include <cmath>
#include "lbgb_fix64.cuh"
using namespace lbgb;
typedef long double LD;
static const int CX[9] = {0, 1, 0, -1, 0, 1, -1, -1, 1}, CY[9] = {0, 0, 1, 0, -1, 1, 1, -1, -1};
extern "C" {
// taken[k]: whether node k is in range; f (n, 9) -> out (n, 9), fields (n, 3)
void collide(const double *f, long n, double omega, double *out, double *fld, unsigned char *taken) {
    fix64::Factor k;
    const bool ok = fix64::omega_factor(omega, k);
    for (long i = 0; i < n; ++i) {
        const double(&x)[9] = *reinterpret_cast<const double(*)[9]>(f + 9 * i);
        double(&o)[9] = *reinterpret_cast<double(*)[9]>(out + 9 * i);
        taken[i] = ok && fix64::collide(x, k, o);
        double &rho = fld[3 * i] = x[0];
        for (int c = 1; c < 9; ++c) rho += x[c];
        if (!fix64::velocity(x, rho, fld[3 * i + 1], fld[3 * i + 2])) taken[i] |= 2;
    }
}
// errors against extended precision: the given results', and an FP64 evaluation's
void errors(const double *f, long n, double omega, const double *out, const double *fld, double *e) {
    for (int j = 0; j < 6; ++j) e[j] = 0;
    for (long i = 0; i < n; ++i, f += 9, out += 9, fld += 3) {
        LD r = 0, jx = (LD)f[1] - f[3] + f[5] - f[6] - f[7] + f[8], jy = (LD)f[2] - f[4] + f[5] + f[6] - f[7] - f[8];
        double dr = 0;
        for (int c = 0; c < 9; ++c) r += f[c], dr += f[c];
        const LD ux = jx / r, uy = jy / r;
        const double dx = (f[1] - f[3] + f[5] - f[6] - f[7] + f[8]) / dr, dy = (f[2] - f[4] + f[5] + f[6] - f[7] - f[8]) / dr;
        for (int c = 0; c < 9; ++c) {
            const LD w = c == 0 ? 4.L / 9 : c < 5 ? 1.L / 9 : 1.L / 36, cu = CX[c] * ux + CY[c] * uy;
            const LD x = f[c] + (LD)omega * (w * r * (1 + 3 * cu + 4.5L * cu * cu - 1.5L * (ux * ux + uy * uy)) - f[c]);
            const double dw = (c == 0 ? 4. / 9 : c < 5 ? 1. / 9 : 1. / 36) * dr, dc = CX[c] * dx + CY[c] * dy;
            const double d = f[c] + omega * (dw * (1 + 3 * dc + 4.5 * dc * dc - 1.5 * (dx * dx + dy * dy)) - f[c]);
            e[1] = fmax(e[1], (double)fabsl(out[c] - x));
            e[2] = fmax(e[2], (double)fabsl(d - x));
        }
        e[4] = fmax(e[4], (double)fmaxl(fabsl(fld[1] - ux), fabsl(fld[2] - uy)));
        e[5] = fmax(e[5], (double)fmaxl(fabsl(dx - ux), fabsl(dy - uy)));
    }
}
long conversions(const double *x, long n, const long long *v, long m) {
    long bad = 0;
    for (long i = 0; i < n; ++i) {
        uint32_t worst = 0;
        const uint64_t y = fix64::to_fix(x[i], 3u, worst);
        bad += worst > fix64::MAX_SHIFT - 3u || y != (uint64_t)(x[i] * 0x1p61);
        if (x[i] >= 0x1p-8) bad += fix64::to_double(y) != x[i];
    }
    for (long i = 0; i < m; ++i) {
        const double exact = (double)((LD)v[i] * 0x1p-61L);  // one rounding, to nearest even
        bad += fix64::to_double_signed(v[i]) != exact;
        if (v[i] >= (1ll << 40)) bad += fix64::to_double((uint64_t)v[i]) != exact;
    }
    return bad;
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fix64")
    (d / "fix64.cpp").write_text(SOURCE)
    so = str(d / "fix64.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "latticeboltzmann_gb300", "csrc"), "-o", so, str(d / "fix64.cpp")], check=True)
    return ctypes.CDLL(so)


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def collide(lib, f, omega):
    f = np.ascontiguousarray(f)
    n = len(f)
    out, fld, taken = np.full((n, 9), np.nan), np.zeros((n, 3)), np.zeros(n, np.uint8)
    lib.collide(ptr(f), ctypes.c_long(n), ctypes.c_double(omega), ptr(out), ptr(fld), ptr(taken))
    return out, fld, taken


def states(n, u, noise, seed):
    rng = np.random.default_rng(seed)
    cx = np.array([0, 1, 0, -1, 0, 1, -1, -1, 1])
    cy = np.array([0, 0, 1, 0, -1, 1, 1, -1, -1])
    w = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
    rho, ux, uy = rng.uniform(0.9, 1.1, (n, 1)), rng.uniform(-u, u, (n, 1)), rng.uniform(-u, u, (n, 1))
    cu = cx * ux + cy * uy
    return w * rho * (1 + 3 * cu + 4.5 * cu ** 2 - 1.5 * (ux ** 2 + uy ** 2)) * (1 + noise * rng.uniform(-1, 1, (n, 9)))


@pytest.mark.parametrize("omega", [0.0, 0.3, 1.0, 1.7, 1.9999])
@pytest.mark.parametrize("u,noise", [(1e-8, 0.0), (0.01, 1e-3), (0.1, 0.05), (0.16, 0.01)])
def test_node_against_extended_precision(lib, omega, u, noise):
    f = states(20000, u, noise, 7)
    out, fld, taken = collide(lib, f, omega)
    assert (taken == 1).all()
    e = np.zeros(6)
    lib.errors(ptr(f), ctypes.c_long(len(f)), ctypes.c_double(omega), ptr(out), ptr(fld), ptr(e))
    if omega > 0:
        assert e[1] < e[2]                  # the FP64 evaluation of the same node
    else:
        assert np.array_equal(out, f)
    assert e[4] <= e[5]
    # mass and momentum change only by the rounding of the stored values
    c = np.array([[1] * 9, [0, 1, 0, -1, 0, 1, -1, -1, 1], [0, 0, 1, 0, -1, 1, 1, -1, -1]], dtype=np.longdouble)
    drift = np.abs((out.astype(np.longdouble) - f) @ c.T)
    assert drift.max() < 9 * 2.0 ** -56


def test_conversions_over_their_range(lib):
    rng = np.random.default_rng(1)
    x = np.ldexp(rng.uniform(0.5, 1, 200000), -rng.integers(0, 20, 200000))
    x = np.concatenate([x, np.ldexp(1.0, -np.arange(1, 21)), np.nextafter(np.ldexp(1.0, -np.arange(0, 20)), 0)])
    v = (rng.integers(-2 ** 62, 2 ** 62, 200000) >> rng.integers(0, 62, 200000)).astype(np.int64)
    edge = np.array([0, 1, -1, 2 ** 32 - 1, 2 ** 32, -2 ** 32, 2 ** 53, 2 ** 53 + 1, 2 ** 53 + 3, 2 ** 54 + 2, 2 ** 54 + 6,
                     2 ** 61 - 1, 2 ** 61, 2 ** 62 - 1, -2 ** 62 + 1], dtype=np.int64)
    v = np.concatenate([v, edge])
    lib.conversions.restype = ctypes.c_long
    assert lib.conversions(ptr(x), ctypes.c_long(len(x)), ptr(v), ctypes.c_long(len(v))) == 0


def test_refused_nodes(lib):
    rest = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
    bad = []
    for v in (-0.1, 0.0, -0.0, np.nan, np.inf, -np.inf, 5e-324, 2.0 ** -23, 1.0, 2.0, 1e300):
        for i in range(9):
            f = rest.copy()
            f[i] = v
            bad.append(f)
    for f in (rest * 0.7, rest * 1.51, rest * 2.0):        # density out of [3/4, 3/2)
        bad.append(f)
    f = rest.copy()
    f[1] += 0.21                                             # momentum
    bad.append(f)
    out, _, taken = collide(lib, np.array(bad), 1.2)
    assert (taken & 1 == 0).all() and np.isnan(out).all()
    assert (taken & 2 == 2).all()
    for omega in (-0.1, 2.0, np.nan, np.inf):
        assert collide(lib, rest[None], omega)[2][0] == 0
    assert collide(lib, rest[None], 1.3)[2][0] == 1
    assert np.array_equal(collide(lib, rest[None], 1.3)[0][0], rest)  # the rest state stays
