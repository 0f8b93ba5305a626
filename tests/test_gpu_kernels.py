"""The kernels at the sizes and values where their forms change: values that
block fixed point leaves to FP64 lines, whole elements per CTA, launches that
start under the one before (small problems) and the others."""
import numpy as np
import pytest

from conftest import dg, max_rel, pressure, workloads

pytestmark = pytest.mark.gpu

RHS_TOL = 1e-12  # one right-hand side: rounding only (tests/test_gpu_parity.py)


def problem(order, ne, precision=64, width=(0.5, 0.5, 0.5), **kw):
    W = workloads()
    cfg = W.gaussian_pulse(seed=3, num_elements=ne, order=order, width=0.5, sponge=1, **kw)
    cfg["ELEMENT_WIDTH"] = list(width)
    cfg["STARTING_CORNER"] = [-0.5 * n * w for n, w in zip(ne, width)]
    cfg["PRECISION"] = precision
    cfg["DT"] = W.cfl_dt(cfg)
    return cfg


def random_state(s, seed, spread=0):
    """Fluxes of both equations of one size, each value times a power of two
    down to 2^-spread."""
    rng = np.random.default_rng(seed)
    rho = rng.standard_normal(s.dims) * 1e-3 * 2.0 ** -rng.integers(0, spread + 1, s.dims)
    vel = rng.standard_normal((3,) + s.dims) * 1e-6 * 2.0 ** -rng.integers(0, spread + 1, (3,) + s.dims)
    return rho, vel


@pytest.mark.parametrize("order", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("spread,width", [(60, (0.5, 0.5, 0.5)), (0, (0.5, 0.2, 0.9))])
def test_rhs_of_uneven_lines_matches_oracle(order, spread, width, oracle_for):
    """Values of one line that differ by up to 2^60, and elements that are no
    cubes (the fixed-point operator is axis 0's, rescaled)."""
    cfg = problem(order, (3, 2, 4), width=width)
    with dg().Solver(cfg) as s:
        o = oracle_for(cfg)
        rho, vel = random_state(s, order, spread)
        s.set_state(rho, vel)
        o.set_state(rho, vel)
        (r, v), (ro, vo) = s.rhs(), o.rhs()
    assert max_rel(r, ro) <= RHS_TOL
    for a in range(3):
        assert max_rel(v[a], vo[a]) <= RHS_TOL


@pytest.mark.parametrize("order", [1, 3, 4, 7])
@pytest.mark.parametrize("exponent", [-900, 900])
def test_lines_outside_fixed_point_scale(order, exponent):
    """With linear fluxes the right-hand side scales with the state.  At
    2^-900 and 2^900 every line's largest value is outside the exponents that
    fixed point takes, so the FP64 lines produce it."""
    cfg = problem(order, (2, 3, 2))
    cfg["B_OVER_A"] = 0.0
    with dg().Solver(cfg) as s:
        rho, vel = random_state(s, 7 * order)
        s.set_state(rho, vel)
        r, v = s.rhs()
        s.set_state(np.ldexp(rho, exponent), np.ldexp(vel, exponent))
        r2, v2 = s.rhs()
    assert max_rel(np.ldexp(r2, -exponent), r) <= RHS_TOL
    assert max_rel(np.ldexp(v2, -exponent), v) <= RHS_TOL


@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_values_spread_as_in_the_oracle(order, bad, oracle_for):
    """A NaN or infinity at one node reaches exactly the nodes it reaches in
    the oracle; the others are what they are without it."""
    cfg = problem(order, (3, 3, 3))
    with dg().Solver(cfg) as s:
        o = oracle_for(cfg)
        rho, vel = random_state(s, order)
        K = order + 1
        rho[K + 1, K, 2 * K - 1] = bad  # a node of the middle element, on two of its faces
        s.set_state(rho, vel)
        o.set_state(rho, vel)
        (r, v), (ro, vo) = s.rhs(), o.rhs()
    for got, want in [(r, ro)] + [(v[a], vo[a]) for a in range(3)]:
        fine = np.isfinite(want)
        assert 0 < np.count_nonzero(~fine) < want.size
        assert np.array_equal(np.isfinite(got), fine)
        assert max_rel(got[fine], want[fine]) <= RHS_TOL


def test_zero_state_stays_zero():
    """Lines of zeros take a path of their own."""
    for order in (1, 3, 4, 5):
        cfg = problem(order, (3, 2, 2))
        with dg().Solver(cfg) as s:
            s.set_state(np.zeros(s.dims), np.zeros((3,) + s.dims))
            s.step(cfg["DT"], 2)
            r, v = s.state()
        assert not r.any() and not v.any()


# FP32 elements per CTA: 16, 7, 4 at orders 1, 2, 3; FP64: 16, 9, 2, 2 at orders 1 to 4
@pytest.mark.parametrize("order,ne", [(1, (1, 1, 1)), (1, (1, 3, 5)), (1, (2, 2, 4)), (1, (1, 1, 17)), (2, (1, 2, 3)),
                                      (2, (1, 1, 7)), (2, (2, 2, 2)), (2, (1, 1, 9)), (2, (1, 2, 5)), (3, (1, 1, 3)),
                                      (3, (2, 2, 1)), (3, (1, 1, 5)), (4, (1, 1, 3)), (5, (1, 2, 1)), (7, (1, 1, 2))])
def test_fp32_partly_filled_blocks_within_tolerance(order, ne):
    """One element less and more than fills a CTA: FP32 against FP64 within the
    form's 1e-5 relative L2."""
    out = []
    for precision in (64, 32):
        cfg = problem(order, ne, precision)
        with dg().Solver(cfg) as s:
            s.step(cfg["DT"], 4)
            out.append(s.state())
    for a, b in zip(out[1], out[0]):
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)


@pytest.mark.parametrize("order,ne", [(1, (47, 47, 46)), (2, (31, 31, 32)), (3, (25, 25, 22))])
def test_fp32_above_the_dependent_launch_rule(order, ne):
    """More than 0.8 M nodes: launches that wait for the one before, at the
    orders whose elements share a CTA."""
    out = []
    for precision in (64, 32):
        cfg = problem(order, ne, precision)
        with dg().Solver(cfg) as s:
            s.step(cfg["DT"], 2)
            out.append(s.state())
    for a, b in zip(out[1], out[0]):
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)


@pytest.mark.parametrize("order,n", [(2, 40), (3, 36), (5, 22)])
def test_batch_blocks_with_several_tiles(order, n):
    """A group with more tiles than blocks beside a tiny one: tiles beyond a
    block's first come from the counter, which the step's last launch resets."""
    m = dg()
    W = workloads()
    cfgs = W.config4(seed=2, n=2)
    for c, k in zip(cfgs, (n, 4)):
        c["ORDER"] = order
        c["NUM_ELEMENTS"] = [k, k, k]
        c["STARTING_CORNER"] = [-0.125 * k, -0.125 * k, 0.0]
        c["DT"] = W.cfl_dt(c)
    with m.Batch(cfgs) as b:
        b.step(2)
        b.step(3)
        got = [b.state(i) for i in range(2)]
    for c, (r, v) in zip(cfgs, got):
        with m.Solver(c) as s:
            s.step(c["DT"], 5)
            r1, v1 = s.state()
        assert np.max(np.abs(r1)) > 0
        assert max_rel(pressure(c, r), pressure(c, r1)) <= 2e-5
        assert max_rel(v, v1) <= 2e-5
