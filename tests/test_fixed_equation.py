"""One equation of a stage line in block fixed point (fix_equation of
csrc/fixed_line.cuh) on the CPU against extended-precision sums: its unit is
that of its own largest value, whatever the other equation's fluxes are, and the
operator is the one given.

Bound, in units u of the output (an eighth of 2^-56 of the largest of the
equation's values times 2^r): 131 u as in tests/test_fixed_line.py, 2 u more
where the rest of a row beyond its mirror image is added from high halves, and
the rounding of the result to double.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, dg

SHIM = r"""
#include "fixed_line.cuh"
using namespace dg;
template <int K>
static int run(const double* rows, int eq, double x, double y, int pm, const double* v, const double* w,
               const double* vo, const double* wo, const double* jump, double* out, int* e_out)
{
    double R[K][K + 2];
    for (int i = 0; i < K; i++)
        for (int j = 0; j < K + 2; j++) R[i][j] = rows[i * (K + 2) + j];
    FixLine<K, 2> L;
    const FixFlux f[2] = {{x, y, pm}, {x, y, pm}};
    if (!fix_axis<K, 2>(R, 1, f, L)) return -1;
    const double a[2] = {vo[0], vo[1]}, b[2] = {wo ? wo[0] : 0.0, wo ? wo[1] : 0.0};
    *e_out = L.e_out[eq];
    return w ? fix_equation<K, true>(L, eq, pm, v, w, 1, a, b, jump[0], jump[1], out)
             : fix_equation<K, false>(L, eq, pm, v, nullptr, 1, a, b, jump[0], jump[1], out);
}
extern "C" int eq_run(int K, const double* rows, int eq, double x, double y, int pm, const double* v, const double* w,
                      const double* vo, const double* wo, const double* jump, double* out, int* e_out)
{
    switch (K) {
    case 2: return run<2>(rows, eq, x, y, pm, v, w, vo, wo, jump, out, e_out);
    case 3: return run<3>(rows, eq, x, y, pm, v, w, vo, wo, jump, out, e_out);
    case 4: return run<4>(rows, eq, x, y, pm, v, w, vo, wo, jump, out, e_out);
    case 5: return run<5>(rows, eq, x, y, pm, v, w, vo, wo, jump, out, e_out);
    case 6: return run<6>(rows, eq, x, y, pm, v, w, vo, wo, jump, out, e_out);
    case 7: return run<7>(rows, eq, x, y, pm, v, w, vo, wo, jump, out, e_out);
    case 8: return run<8>(rows, eq, x, y, pm, v, w, vo, wo, jump, out, e_out);
    }
    return -2;
}
"""
q = np.longdouble


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("eq")
    src, so = d / "shim.cpp", d / "libshim.so"
    src.write_text(SHIM)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-w", "-shared", "-fPIC",
                           "-I" + os.path.join(ROOT, "3ddg_gb300", "csrc"), str(src), "-o", str(so)])
    lib = C.CDLL(str(so))
    lib.eq_run.argtypes = [C.c_int, C.c_void_p, C.c_int, C.c_double, C.c_double, C.c_int] + [C.c_void_p] * 7
    return lib


def evaluate(lib, K, rows, eq, x, y, pm, v, w, vo, wo, jump):
    out, e_out = np.empty(K), np.zeros(1, dtype=np.int32)
    p = lambda a: None if a is None else a.ctypes.data_as(C.c_void_p)  # noqa: E731
    rc = lib.eq_run(K, p(rows), eq, x, y, pm, p(v), p(w), p(vo), p(wo), p(jump), p(out), p(e_out))
    return rc, out, int(e_out[0])


def exact(K, rows, x, y, v, w, vo, wo, jump):
    r = rows.astype(q)
    s = v.astype(q) + (0 if w is None else w.astype(q))
    o = vo.astype(q) + (0 if w is None else wo.astype(q))
    f0 = q(x) * (o[0] + s[0]) + q(y) * q(jump[0])
    fN = -q(x) * (o[1] + s[-1]) + q(y) * q(jump[1])
    return r[:, :K] @ s + r[:, K] * f0 + r[:, K + 1] * fN


def rows_of(K, scale):
    ops = dg().line_operators(K - 1)
    return np.ascontiguousarray(np.column_stack([ops["deriv"] * scale, ops["lift0"], ops["liftN"]]))


def mirrored(K, rows):
    m, h = rows.copy(), K // 2
    m[K - h:, :K] = -m[:h, :K][::-1, ::-1]
    m[:, K + 1] = m[::-1, K]
    if K % 2:
        m[h, h] = 0.0
        m[h, K - h:K] = -m[h, :h][::-1]
    return m


def draw(rng, K, size, spread, two):
    one = lambda n: size * rng.standard_normal(n) * 2.0 ** -rng.integers(0, spread + 1, n)  # noqa: E731
    v, vo = one(K), one(2)
    w, wo = (one(K) * 1e-3, one(2) * 1e-3) if two else (None, None)
    return v, w, vo, wo


def unit(v, w, vo, wo, jump, pm, e_out):
    """u from the equation's own largest value."""
    top = max(float(np.max(np.abs(a))) for a in (v, w, vo, wo, np.ldexp(jump, -pm)) if a is not None)
    return q(2.0) ** (int(np.frexp(top)[1]) + 1022 + e_out - 1085)


@pytest.mark.parametrize("K", range(2, 9))
@pytest.mark.parametrize("two", [False, True])
def test_unit_is_the_equations_own(K, two, shim):
    """Jumps of the other equation from far below to far above the line's own
    values (as scaled by 2^pm)."""
    rng = np.random.default_rng(100 * K + two)
    for trial in range(300):
        scale = float(10.0 ** rng.uniform(-6, 2))
        rows = rows_of(K, scale) if K not in (2, 3, 5) else mirrored(K, rows_of(K, scale))
        pm = int(rng.integers(-12, 13))
        x, y = 0.5 * scale, float(0.5 * scale * 2.0 ** -pm * rng.uniform(0.6, 1.5))
        size = 2.0 ** rng.integers(-600, 600)
        v, w, vo, wo = draw(rng, K, size, int(rng.choice([0, 1, 8, 40])), two)
        jump = np.ldexp(size * rng.standard_normal(2), pm - int(rng.integers(-60, 61)))
        jump[rng.random(2) < 0.2] = 0.0
        rc, out, e_out = evaluate(shim, K, rows, trial % 2, x, y, pm, v, w, vo, wo, jump)
        assert rc == 1
        want = exact(K, rows, x, y, v, w, vo, wo, jump)
        u = unit(v, w, vo, wo, jump, pm, e_out)
        err = np.abs(out.astype(q) - want)
        assert np.all(err <= 131 * u + np.abs(want) * q(2.0 ** -53)), (trial, err / u)


@pytest.mark.parametrize("K", range(2, 9))
@pytest.mark.parametrize("off", [1e-14, 5e-13])
def test_operator_is_the_given_one(K, off, shim):
    """Rows and lift columns whose mirror symmetry is broken by more than
    rounding and less than 1e-12."""
    rng = np.random.default_rng(1000 * K)
    for trial in range(200):
        rows = mirrored(K, rows_of(K, 0.01))
        top = [np.max(np.abs(rows[:, :K])), np.max(np.abs(rows[:, K:]))]
        for j in range(K + 2):
            rows[:, j] += off * top[j >= K] * rng.uniform(-0.5, 0.5, K)
        x, y, pm = 0.005, 0.004, 0
        v, w, vo, wo = draw(rng, K, 1.0, int(rng.choice([0, 8])), bool(trial % 2))
        jump = rng.standard_normal(2)
        rc, out, e_out = evaluate(shim, K, rows, 0, x, y, pm, v, w, vo, wo, jump)
        assert rc == 1
        want = exact(K, rows, x, y, v, w, vo, wo, jump)
        u = unit(v, w, vo, wo, jump, pm, e_out)
        err = np.abs(out.astype(q) - want)
        assert np.all(err <= 133 * u + np.abs(want) * q(2.0 ** -53)), (trial, err / u)


@pytest.mark.parametrize("K", range(2, 9))
@pytest.mark.parametrize("lumped", [False, True])
def test_library_operators_within_solver_rounding(K, lumped, shim):
    """The library's D and lift columns as they are: applied as given, or (K =
    2, 3, 5) with rows that differ from them by no more than 2^-48 of the
    largest entry, the rounding of the solve that produced them."""
    rng = np.random.default_rng(K)
    ops = dg().line_operators(K - 1, lumped=lumped)
    rows = np.ascontiguousarray(np.column_stack([ops["deriv"] * 0.01, ops["lift0"], ops["liftN"]]))
    noise = 2.0 ** -48 if K in (2, 3, 5) else 0.0
    x, y, pm = 0.005, 0.004, 0
    for _ in range(200):
        v, w, vo, wo = draw(rng, K, 1.0, 0, True)
        jump = rng.standard_normal(2)
        rc, out, e_out = evaluate(shim, K, rows, 0, x, y, pm, v, w, vo, wo, jump)
        assert rc == 1
        want = exact(K, rows, x, y, v, w, vo, wo, jump)
        f = [x * (vo[0] + wo[0] + v[0] + w[0]) + y * jump[0], -x * (vo[1] + wo[1] + v[-1] + w[-1]) + y * jump[1]]
        slack = noise * (np.max(np.abs(rows[:, :K])) * np.sum(np.abs(v + w)) +
                         np.max(np.abs(rows[:, K:])) * np.sum(np.abs(f)))
        err = np.abs(out.astype(q) - want)
        assert np.all(err <= 133 * unit(v, w, vo, wo, jump, pm, e_out) + slack + np.abs(want) * q(2.0 ** -53))


@pytest.mark.parametrize("K", range(2, 9))
@pytest.mark.parametrize("two", [False, True])
def test_zeros_and_what_is_left_to_fp64(K, two, shim):
    """Lines of +-0 give +0; one denormal, huge or non-finite value anywhere
    leaves the line to the caller, untouched."""
    rows = rows_of(K, 0.01)

    def line(fill):
        v, vo, jump = np.full(K, fill), np.full(2, fill), np.full(2, fill)
        return v, np.full(K, fill) if two else None, vo, np.full(2, fill) if two else None, jump

    for fill in (0.0, -0.0):
        rc, out, _ = evaluate(shim, K, rows, 0, 0.005, 0.004, 0, *line(fill))
        assert rc == 1 and not out.any() and not np.signbit(out).any()
    for bad in (5e-324, -1e-310, 2.0 ** -900, 2.0 ** 900, np.inf, np.nan):
        for which in range(5):
            for fill in (0.0, 1.0) if abs(bad) > 1 or bad != bad else (0.0,):
                a = line(fill)
                if a[which] is None:
                    continue
                a[which][-1] = bad
                rc, _, _ = evaluate(shim, K, rows, 0, 0.005, 0.004, 0, *a)
                assert rc == 0, (bad, which, fill)
