"""Right-hand sides against extended-precision sums of the operator in use:
states whose momentum and mass fluxes are of very different size, and operators
from matrix files whose mirror symmetry is broken a little (the fixed-point
kernels apply what row K-1-i has beyond the mirror image of row i) or more (the
FP64 kernels of dg_kernels.cuh).

Bound: with T the sum over axes of (largest operator row sum) x (largest value
of the equation's own terms), a fixed-point sum is off by at most 131 of its
units, 17 x 2^-53 T per axis, and a chain of K + 6 FP64 operations by at most
14 x 2^-53 T; with the fluxes, the stage combination and LDG's two levels,
64 x 2^-53 T.
"""
import ctypes as C
import os

import numpy as np
import pytest

from conftest import dg, max_rel, workloads

pytestmark = pytest.mark.gpu

q = np.longdouble
EPS = 64 * 2.0 ** -53


class Reference:
    """The semi-discrete scheme of one block of ``ne`` elements in extended
    precision, zero outside non-periodic faces, and per equation the T of the
    bound above.  Numerical fluxes by the jumps of the other equation's flux."""

    def __init__(self, cfg, ops):
        self.cfg, self.K, self.ne = cfg, cfg["ORDER"] + 1, cfg["NUM_ELEMENTS"]
        self.D, self.L0, self.LN = (ops[k].astype(q) for k in ("deriv", "lift0", "liftN"))
        self.row = float(np.max(np.abs(self.D).sum(1) + np.abs(self.L0) + np.abs(self.LN)))

    def split(self, g):
        K, (X, Y, Z) = self.K, self.ne
        return g.astype(q).reshape(-1, X, K, Y, K, Z, K).transpose(0, 1, 3, 5, 2, 4, 6)

    def join(self, u):
        K, (X, Y, Z) = self.K, self.ne
        return u.transpose(0, 1, 4, 2, 5, 3, 6).reshape(-1, X * K, Y * K, Z * K)

    def along(self, v, a):
        return np.moveaxis(np.moveaxis(v, 3 + a, -1) @ self.D.T, -1, 3 + a)

    def ends(self, v, a):
        lo, hi = np.take(v, 0, axis=3 + a), np.take(v, self.K - 1, axis=3 + a)
        left, right = np.roll(hi, 1, a), np.roll(lo, -1, a)
        if not self.cfg["BC_IS_PERIODIC"][a]:
            s = [slice(None)] * 5
            s[a] = 0
            left[tuple(s)] = 0
            s[a] = self.ne[a] - 1
            right[tuple(s)] = 0
        return lo, hi, left, right

    def lift(self, g0, gN, a):
        shape = [1] * 6
        shape[3 + a] = self.K
        return self.L0.reshape(shape) * np.expand_dims(g0, 3 + a) + self.LN.reshape(shape) * np.expand_dims(gN, 3 + a)

    def rhs(self, rho, vel, sigma):
        c = self.cfg
        c0, r0, ba, Dc = (q(c[k]) for k in ("C0", "RHO0", "B_OVER_A", "DIFF_CONST"))
        u, sig = self.split(np.concatenate([rho[None], vel])), self.split(sigma[None])[0]
        d = u[0]
        size = [0.0, 0.0, 0.0, 0.0]
        out = [np.zeros_like(d)]
        fm = c0 * c0 / r0 * (d + ba / (2 * r0) * d * d)
        for a in range(3):
            w = q(c["ELEMENT_WIDTH"][a])
            fa = u[1 + a] * (r0 if ba == 0 else d + r0)
            m0, mN, ml, mr = self.ends(fm, a)
            a0, aN, al, ar = self.ends(fa, a)
            k, g = c0 / (2 * r0), r0 / (2 * c0)
            out.append((self.along(fm, a) + self.lift((ml + m0) / 2 + k * (al - a0),
                                                      -((mr + mN) / 2 + k * (aN - ar)), a)) / w)
            f = self.along(fa, a) + self.lift((al + a0) / 2 + g * (ml - m0), -((ar + aN) / 2 + g * (mN - mr)), a)
            most = lambda *v: max(float(np.max(np.abs(x))) for x in v)  # noqa: E731
            size[1 + a] += self.row * most(fm, k * (al - a0), k * (aN - ar)) / float(w)
            size[0] += self.row * most(fa, g * (ml - m0), g * (mN - mr)) / float(w)
            if c["EVALUATE_DIFFUSION"]:
                d0, dN, dl, dr = self.ends(d, a)
                G = (self.along(d, a) + self.lift((dl + d0) / 2, -(dr + dN) / 2, a)) * (Dc / w)
                q0, qN, ql, qr = self.ends(G, a)
                f = f + self.along(G, a) + self.lift((ql + q0) / 2, -(qr + qN) / 2, a)
                size[0] += self.row * most(G) / float(w)
                size[0] += self.row * self.row * float(Dc) * most(d) / float(w) ** 2
            out[0] = out[0] + f / w
        top = float(np.max(np.abs(sig)))
        size = [s + top * float(np.max(np.abs(u[i]))) for i, s in enumerate(size)]
        return self.join(np.stack(out) - sig * u), size


def problem(order, ne=(3, 2, 4), periodic=(0, 0, 0), **kw):
    cfg = workloads().gaussian_pulse(seed=5, num_elements=ne, order=order, width=0.5, sponge=1, periodic=periodic, **kw)
    cfg["DT"] = workloads().cfl_dt(cfg)
    return cfg


def acoustic_state(dims, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(dims) * 1e-3, rng.standard_normal((3,) + tuple(dims)) * 1e-6


def check(cfg, ops, s, rho, vel, fields=range(4)):
    _, sigma = s.grid()
    s.set_state(rho, vel)
    r, v = s.rhs()
    want, size = Reference(cfg, ops).rhs(rho, vel, sigma)
    got = np.concatenate([r[None], v])
    for f in fields:
        err = float(np.max(np.abs(got[f].astype(q) - want[f])))
        assert err <= EPS * size[f], (f, err / size[f])


# ----------------------------------------------------- fluxes of uneven size
@pytest.mark.parametrize("order", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("size", [1e-4, 1e-8, 1e-12, 1e-18])
def test_momentum_of_small_densities_beside_large_velocities(order, size):
    """A uniform flow that carries a density disturbance far below a sound
    wave's: the momentum equation sees the disturbance alone (linear fluxes:
    the mass flux has no jumps) and keeps its precision."""
    cfg = problem(order, periodic=(1, 1, 1))
    cfg["B_OVER_A"], cfg["EVALUATE_SPONGE"], cfg["BC_SPONGE_WIDTH"] = 0.0, 0, [0] * 6
    with dg().Solver(cfg) as s:
        rho, vel = acoustic_state(s.dims, order)
        rho *= size * 1e3
        for a in range(3):
            vel[a] = 3.3e-4 * (a + 1)
        check(cfg, dg().line_operators(order), s, rho, vel, (1, 2, 3))


@pytest.mark.parametrize("order", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("size", [1e-4, 1e-8, 1e-12, 1e-18])
def test_mass_of_small_velocities_in_a_large_density(order, size):
    """The reverse: a uniform density, whose momentum flux has no jumps, and a
    velocity field far below a sound wave's."""
    cfg = problem(order, periodic=(1, 1, 1), diffusion=False)
    cfg["B_OVER_A"], cfg["EVALUATE_SPONGE"], cfg["BC_SPONGE_WIDTH"] = 0.0, 0, [0] * 6
    with dg().Solver(cfg) as s:
        rho, vel = acoustic_state(s.dims, order)
        rho[:] = 0.22
        vel *= size * 330.0
        check(cfg, dg().line_operators(order), s, rho, vel, (0,))


# ------------------------------------------------- operators from matrix files
def operator_files(folder, order, off):
    """Matrix and coefficient files whose S of ``order`` has one entry scaled by
    1 + off."""
    import refinputs
    refinputs.write_coeff_files(str(folder))
    path = os.path.join(str(folder), "matrices.txt")
    with open(path, "w") as f:
        for N in range(1, refinputs.KMAX):
            M, S = (np.array(m, dtype=np.float64) for m in refinputs.unit_matrices(N, False))
            if N == order:
                S[0, 1] *= 1.0 + off
            f.write("Order=%d\n" % N)
            for r in np.concatenate([M, S]):
                f.write(" ".join(refinputs.hexd(v) for v in r) + "\n")
    return path, os.path.join(str(folder), "hardcoded_coeff.txt")


def asymmetry(ops):
    D = ops["deriv"]
    return float(np.max(np.abs(D + D[::-1, ::-1])) / np.max(np.abs(D)))


def noalloc_rhs(cfg, ops, s, ne):
    """dg_eval_rhs_noalloc of a Solver's state with the caller's M and S."""
    import torch
    m = dg()
    K = cfg["ORDER"] + 1
    base, NP, n_elem = s.device_state()
    index = np.arange(n_elem).reshape(ne)
    nbr = np.empty(tuple(ne) + (6,), dtype=np.int32)
    for a in range(3):
        for side in (0, 1):
            n = np.roll(index, -1 if side else 1, a).copy()
            edge = [slice(None)] * 3
            edge[a] = ne[a] - 1 if side else 0
            if not cfg["BC_IS_PERIODIC"][a]:
                n[tuple(edge)] = -1
            nbr[..., 2 * a + side] = n
    _, sig = s.grid()
    d_nbr = torch.from_numpy(nbr.reshape(-1, 6)).cuda()
    d_sig = torch.from_numpy(sig[::K, ::K, ::K].reshape(-1).copy()).cuda()
    d_rhs = torch.full((4 * n_elem * NP,), float("nan"), dtype=torch.float64, device="cuda")
    mass, stiff = (np.ascontiguousarray(ops[k]) for k in ("mass", "stiff"))
    s.synchronize()
    torch.cuda.synchronize()
    rc = m.lib().dg_eval_rhs_noalloc(C.byref(s.params), mass.ctypes.data, stiff.ctypes.data, base[0],
                                     d_nbr.data_ptr(), d_sig.data_ptr(), d_rhs.data_ptr(), n_elem, None)
    assert rc == 0, m.lib().dg_last_error().decode()
    torch.cuda.synchronize()
    X, Y, Z = ne
    g = d_rhs.cpu().numpy().reshape(4, X, Y, Z, NP)[..., :K ** 3].reshape(4, X, Y, Z, K, K, K)
    return g.transpose(0, 1, 4, 2, 5, 3, 6).reshape(4, X * K, Y * K, Z * K)


@pytest.mark.parametrize("order", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("diffusion", [True, False])
def test_operator_slightly_off_mirror_symmetry(order, diffusion, tmp_path):
    """An operator off by more than rounding and less than the 1e-12 that the
    fixed-point kernels take is applied as given, by the handle and by
    dg_eval_rhs_noalloc."""
    mf, cf = operator_files(tmp_path, order, 4e-13)
    ops = dg().line_operators(order, matrix_file=mf, coeff_file=cf)
    assert 2e-14 < asymmetry(ops) <= 1e-12
    ne = (3, 2, 4)
    cfg = problem(order, ne, diffusion=diffusion)
    cfg["B_OVER_A"] = 0.0
    with dg().Solver(cfg, mf, cf) as s:
        rho, vel = acoustic_state(s.dims, order)
        check(cfg, ops, s, rho, vel)
        s.set_state(rho, vel)
        got = noalloc_rhs(cfg, ops, s, ne)
        want, size = Reference(cfg, ops).rhs(rho, vel, s.grid()[1])
    for f in range(4):
        assert float(np.max(np.abs(got[f].astype(q) - want[f]))) <= EPS * size[f]


# 9 elements: the last block of the FP64 kernels (4 or 2 elements at orders 1 to 3) is partly filled
@pytest.mark.parametrize("order", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("diffusion", [True, False])
def test_operator_without_mirror_symmetry(order, diffusion, tmp_path):
    """The FP64 kernels of dg_kernels.cuh, by the handle and by
    dg_eval_rhs_noalloc (which copies the operators into its scratch and clears
    its boundary flags for them)."""
    mf, cf = operator_files(tmp_path, order, 1e-6)
    ops = dg().line_operators(order, matrix_file=mf, coeff_file=cf)
    assert asymmetry(ops) > 1e-7
    ne = (1, 3, 3)
    cfg = problem(order, ne, diffusion=diffusion)
    with dg().Solver(cfg, mf, cf) as s:
        rho, vel = acoustic_state(s.dims, order)
        check(cfg, ops, s, rho, vel)
        s.set_state(rho, vel)
        got = noalloc_rhs(cfg, ops, s, ne)
        want, size = Reference(cfg, ops).rhs(rho, vel, s.grid()[1])
    for f in range(4):
        assert float(np.max(np.abs(got[f].astype(q) - want[f]))) <= EPS * size[f]


@pytest.mark.parametrize("order", [1, 2, 4, 7])
@pytest.mark.parametrize("off", [0.0, 4e-13, 1e-6])
def test_step_and_download_of_any_operator(order, off, tmp_path):
    """step_state_async against step and state, bit for bit; once the fluxes of
    the state are there, the last stage writes the host order itself (no launch
    beyond the step's)."""
    import torch
    mf, cf = operator_files(tmp_path, order, off)
    cfg = problem(order, (2, 3, 3))
    with dg().Solver(cfg, mf, cf) as a, dg().Solver(cfg, mf, cf) as b:
        rho, vel = acoustic_state(a.dims, order)
        for s in (a, b):
            s.set_state(rho, vel)
            s.step(cfg["DT"], 1)
        pin = lambda n: torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()  # noqa: E731
        out = pin(tuple(a.dims)), pin((3,) + tuple(a.dims))
        before = a.launches
        a.step(cfg["DT"], 1)
        per_step = a.launches - before
        before = b.launches
        b.step_state_async(cfg["DT"], *out)
        assert b.launches - before == per_step
        b.synchronize()
        r, v = a.state()
        assert np.any(r) and np.array_equal(out[0], r) and np.array_equal(out[1], v)


@pytest.mark.parametrize("precision,off", [(64, 0.0), (64, 1e-6), (32, 0.0)])
def test_operators_follow_dt(precision, off, tmp_path):
    """Steps of changing dt, the right-hand side before the first of them and
    between them, against the oracle with the same operator."""
    import pyoracle
    import refinputs
    order = 3
    mf, cf = operator_files(tmp_path, order, off)
    cfg = problem(order, (3, 2, 4))
    cfg["PRECISION"] = precision
    o = pyoracle.Oracle(dict(cfg, PRECISION=64), *refinputs.read_matrices(mf, order), refinputs.read_zeros(cf, order))
    tol = 1e-10 if precision == 64 else 1e-5
    with dg().Solver(cfg, mf, cf) as s:
        for k, f in enumerate((1.0, 0.5, 0.5, 0.75)):
            if k != 1:
                (r, v), (ro, vo) = s.rhs(), o.rhs()
                assert max_rel(r, ro) <= tol and max_rel(v, vo) <= tol
            s.step(f * cfg["DT"], 2)
            o.run(f * cfg["DT"], 2)
        (r, v), (ro, vo) = s.state(), o.state()
    assert max_rel(r, ro) <= tol and max_rel(v, vo) <= tol
