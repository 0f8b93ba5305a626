"""The block fixed-point line operator (csrc/fixed_line.cuh) on the CPU against
extended-precision sums, at every order, over magnitudes that differ by many
orders along a line, with zeros, denormals and the largest exponents it takes.

Bound, in units u of the output (an eighth of 2^-56 of the line's largest value
times 2^r, r at most 4.04 row sums): an operand is a sum of at most 8 values
truncated by less than 8 u each and the coefficients of one output sum to less
than 1 (64 u), a product drops at most 2^31 2^27 of the 2^56 that make one u
(n/2 x 8 < 32 u for 8 products), a coefficient is rounded by 2^-60 (n x 8
values x 8/16 u < 32 u), two sums are floored and one is complemented (3 u):
131 u, plus the rounding of the result to double.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, dg

SHIM = r"""
#include "fixed_line.cuh"
#include <algorithm>
using namespace dg;
template <int K>
static int run(const double* rows, int sig, double x, double y, int pm, int swap, const double* v, const double* X,
               const double* Y, double* out, double* unit)
{
    double R[K][K + 2];
    for (int i = 0; i < K; i++)
        for (int j = 0; j < K + 2; j++) R[i][j] = rows[i * (K + 2) + j];
    FixLine<K, 2> L;
    const FixFlux f[2] = {{x, y, pm}, {x, y, pm}};
    if (!fix_axis<K, 2>(R, sig, f, L)) return -1;
    int top = 0;
    for (int j = 0; j < K; j++) top = std::max(top, fix_abs_hi(v[j]));
    for (int s = 0; s < 2; s++) top = std::max(top, fix_abs_hi(X[s]));
    int E = top >> 20, ty = 0;
    for (int s = 0; s < 2; s++) ty = std::max(ty, fix_abs_hi(Y[s]) >> 20);
    if (sig > 0) E = std::max(E, ty - pm);
    if (E < kFixMinExp || E > kFixMaxExp) return 1;
    FixVal xv[K];
    const FixVal none = {0, 0};
    for (int j = 0; j < K; j++) xv[j] = fix_from(v[j], E);
    fix_line<K, 2>(L, 0, xv, fix_from(X[0], E), fix_from(X[1], E), sig > 0 ? fix_from(Y[0], E + pm) : none,
                         sig > 0 ? fix_from(Y[1], E + pm) : none,
                         [&](int i, long long o) {
                             out[i] = fix_to(o, E + L.e_out[0]);
                             out[K + i] = fix_to_fp64(o, E + L.e_out[0]);
                         });
    *unit = std::ldexp(1.0, E + L.e_out[0] - 1085);
    return 0;
}
extern "C" int fix_run(int K, const double* rows, int sig, double x, double y, int pm, const double* v,
                       const double* X, const double* Y, double* out, double* unit)
{
    switch (K) {
    case 2: return run<2>(rows, sig, x, y, pm, 0, v, X, Y, out, unit);
    case 3: return run<3>(rows, sig, x, y, pm, 0, v, X, Y, out, unit);
    case 4: return run<4>(rows, sig, x, y, pm, 0, v, X, Y, out, unit);
    case 5: return run<5>(rows, sig, x, y, pm, 0, v, X, Y, out, unit);
    case 6: return run<6>(rows, sig, x, y, pm, 0, v, X, Y, out, unit);
    case 7: return run<7>(rows, sig, x, y, pm, 0, v, X, Y, out, unit);
    case 8: return run<8>(rows, sig, x, y, pm, 0, v, X, Y, out, unit);
    }
    return -2;
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("fix")
    src, so = d / "shim.cpp", d / "libshim.so"
    src.write_text(SHIM)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-w", "-shared", "-fPIC",
                           "-I" + os.path.join(ROOT, "3ddg_gb300", "csrc"), str(src), "-o", str(so)])
    lib = C.CDLL(str(so))
    lib.fix_run.argtypes = [C.c_int, C.c_void_p, C.c_int, C.c_double, C.c_double, C.c_int] + [C.c_void_p] * 5
    return lib


def call(lib, K, rows, sig, x, y, pm, v, X, Y):
    out, unit = np.empty((2, K)), np.empty(1)  # by either conversion
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    rc = lib.fix_run(K, p(rows), sig, x, y, pm, p(v), p(X), p(Y), p(out), p(unit))
    return rc, out, float(unit[0])


def rows_of(K, scale, sig):
    ops = dg().line_operators(K - 1)
    D, L0 = ops["deriv"] * scale, ops["lift0"]
    LN = ops["liftN"]
    if K in (2, 3, 5):  # rows i < K/2 stand for their mirror images
        h = K // 2
        D[K - h:] = -D[:h][::-1, ::-1]
        if K % 2:
            D[h, h] = 0.0
            D[h, K - h:] = -D[h, :h][::-1]
        LN = L0[::-1]
    return np.ascontiguousarray(np.column_stack([D, L0, sig * LN]))


@pytest.mark.parametrize("K", range(2, 9))
@pytest.mark.parametrize("sig", [1, -1])
def test_line_against_extended_precision(K, sig, shim):
    rng = np.random.default_rng(10 * K + sig)
    for trial in range(400):
        scale = float(10.0 ** rng.uniform(-8, 3))
        rows = rows_of(K, scale, sig)
        # the kernels' proportions: fluxes half of D's scale, Y scaled by 2^pm
        pm = int(rng.integers(-12, 13))
        x, y = 0.5 * scale, float(0.5 * scale * 2.0 ** -pm * rng.uniform(0.6, 1.5))
        size = 2.0 ** rng.integers(-700, 700)
        spread = rng.choice([0, 1, 8, 40, 300])
        draw = lambda n: size * rng.standard_normal(n) * 2.0 ** -rng.integers(0, spread + 1, n)  # noqa: E731
        v, X, Y = draw(K), draw(2), np.ldexp(draw(2), pm)
        for a in (v, X, Y):
            a[rng.random(len(a)) < 0.15] = rng.choice([0.0, -0.0, 5e-324, size])
        if sig < 0:
            x, y, Y = 1.0, 0.0, np.zeros(2)
        rc, out, unit = call(shim, K, rows, sig, x, y, -pm if sig > 0 else 0, v, X, Y)
        assert rc in (0, 1)
        if rc == 1:  # all zeros and denormals
            assert max(np.max(np.abs(v)), np.max(np.abs(X)), np.max(np.abs(np.ldexp(Y, -pm)))) < 2.0 ** -800
            continue
        q = np.longdouble
        r = rows.astype(q)
        f0 = q(x) * q(X[0]) + q(y) * q(Y[0])
        fN = q(-x if sig > 0 else x) * q(X[1]) + q(y) * q(Y[1])
        want = r[:, :K] @ v.astype(q) + r[:, K] * f0 + r[:, K + 1] * fN
        err = np.abs(out.astype(q) - want)
        assert np.all(err <= 131 * q(unit) + np.abs(want) * q(2.0 ** -53)), (trial, err / q(unit))


@pytest.mark.parametrize("K", [2, 5, 8])
def test_line_error_below_fp64_sums(K, shim):
    """Over random lines the largest and the mean error are below those of the
    same sums in FP64."""
    rng = np.random.default_rng(K)
    rows = rows_of(K, 0.01, 1)
    q = np.longdouble
    worst, mean = np.zeros(2), np.zeros(2)
    for _ in range(500):
        v, X, Y = rng.standard_normal(K), rng.standard_normal(2), rng.standard_normal(2)
        rc, out, _ = call(shim, K, rows, 1, 0.005, 0.005, 0, v, X, Y)
        assert rc == 0
        r = rows.astype(q)
        f = [q(0.005) * (q(X[0]) + q(Y[0])), q(0.005) * (q(Y[1]) - q(X[1]))]
        want = r[:, :K] @ v.astype(q) + r[:, K] * f[0] + r[:, K + 1] * f[1]
        s = rows[:, K] * (0.005 * X[0] + 0.005 * Y[0]) + rows[:, K + 1] * (-0.005 * X[1] + 0.005 * Y[1])
        for j in range(K):
            s = s + rows[:, j] * v[j]
        for k, got in enumerate((out, s)):
            e = np.abs(got.astype(q) - want) / np.max(np.abs(want))
            worst[k] = max(worst[k], float(e.max()))
            mean[k] += float(e.mean())
    assert worst[0] <= worst[1] and mean[0] < mean[1]


def test_unusual_operators_are_refused(shim):
    K = 5
    rows = rows_of(K, 1.0, 1)
    v, z = np.ones(K), np.ones(2)
    assert call(shim, K, rows, 1, 0.5, 0.5, 0, v, z, z)[0] == 0
    bad = rows.copy()
    bad[0, 1] *= 1 + 1e-6
    assert call(shim, K, bad, 1, 0.5, 0.5, 0, v, z, z)[0] == -1
    for s in (2.0 ** -100, 2.0 ** 100, np.nan, np.inf):
        assert call(shim, K, rows * s, 1, 0.5, 0.5, 0, v, z, z)[0] == -1
    for w in (np.inf, -np.inf, np.nan, 1e300, 1e-300):
        assert call(shim, K, rows, 1, 0.5, 0.5, 0, np.array([1, w, 1, 1, 1.0]) if abs(w) > 1 or w != w else v * w, z * (w if w == 1e-300 else 1), z * (w if w == 1e-300 else 1))[0] == 1
    zero = rows * 0.0
    rc, out, _ = call(shim, K, zero, 1, 0.0, 0.0, 0, v, z, z)
    assert rc == 0 and np.all(out == 0.0)
