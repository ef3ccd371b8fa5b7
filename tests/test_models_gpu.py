"""Device models and diagnostics against the oracle: Smagorinsky eddy
viscosity (subgrid.f90:609-730), LES steps, z-averaged statistics and Cf
(statistics.f90:26-201), the equilibrium law of the wall solved by Newton
(wallmodel.f90:1951-1985, Newton_solver.f90), and the laminar skin friction
of config 1 against the Blasius value 0.664/sqrt(Re_x)."""
import numpy as np
import pytest

import oracle
from blgpu import cases, FP64, MIXED

pytestmark = pytest.mark.gpu


def rel(a, b):
    nb = np.linalg.norm(b)
    return np.linalg.norm(a - b) / (nb if nb > 0 else 1.0)


def noisy(nx, ny, nz, seed, amp, **kw):
    c = cases.laminar_case(nx=nx, ny=ny, nz=nz, lx=20.0, ly=5.0, lz=3.0, **kw)
    rng = np.random.default_rng(seed)
    c.U = np.asfortranarray(c.U + amp * rng.standard_normal(c.U.shape))
    c.V = np.asfortranarray(c.V + amp * rng.standard_normal(c.V.shape))
    c.W = np.asfortranarray(c.W + amp * rng.standard_normal(c.W.shape))
    return c


@pytest.mark.parametrize("grid", [(26, 14, 11), (60, 17, 15)])
def test_smagorinsky_matches_oracle(gpu, grid):
    c = noisy(*grid, seed=21, amp=0.05)
    s = cases.solver_for(c, les_model=1)
    o = oracle.oracle_for(c)
    nut = s.compute_eddy_viscosity()
    ref = o.smagorinsky()
    inner = (slice(1, -1), slice(1, -1), slice(1, -1))
    assert np.abs(nut[inner] - ref[inner]).max() <= 1e-14 * np.abs(ref).max()
    assert (nut[inner] >= 0).all() and ref.max() > 0
    s.close()


@pytest.mark.parametrize("grid", [(5, 4, 5), (33, 9, 17), (34, 10, 18), (65, 8, 33)])
def test_smagorinsky_tile_edges(gpu, grid):
    """Column kernel at its tile edges: the smallest box, 32 interior columns
    and one more, 8 rows and one more, z chunks of 16 planes and one more (17
    and 32 interior planes).  FP64 repeats the oracle's expressions; FP32
    forms some 40 rounded operations from differences of O(1) velocities
    (each 6e-8 of |u|, over the smallest spacing)."""
    c = noisy(*grid, seed=sum(grid), amp=0.05)
    ref = oracle.oracle_for(c).smagorinsky()
    inner = (slice(1, -1), slice(1, -1), slice(1, -1))
    h = min(np.diff(a).min() for a in (c.x, c.y, c.z))
    for prec in (FP64, MIXED):
        s = cases.solver_for(c, precision=prec, les_model=1)
        nut = s.compute_eddy_viscosity()
        if prec == FP64:
            tol = 1e-14 * np.abs(ref).max()
        else:  # (Cs Delta)^2 times the strain's rounding, 4 differences of two rounded values
            tol = 40 * 6e-8 * np.abs(ref).max() + 8 * 6e-8 / h * 0.11 ** 2 * np.diff(c.y).max() ** (2 / 3) * (
                np.diff(c.x).min() * np.diff(c.z).min()) ** (2 / 3)
        assert np.abs(nut[inner] - ref[inner]).max() <= tol
        s.close()


def test_smagorinsky_of_infinite_quotients(gpu):
    """A state near overflow, as a run leaves it that has blown up: where the
    source's quotient (u_a - u_b)/dx is an infinity the viscosity is one too,
    not a NaN, and the cells whose corner averages add infinities of both signs
    hold NaN as the source's do.  The large velocities overflow over every
    spacing (all below 0.8) in the precision at hand: 1.7e308 in FP64 and 3e38
    in FP32, whose other cells match to FP32's range."""
    grid = (12, 9, 14)
    c = cases.laminar_case(nx=grid[0], ny=grid[1], nz=grid[2], lx=5.0, ly=3.0, lz=5.0)
    assert max(np.diff(a).max() for a in (c.x, c.y, c.z)) < 0.8

    def state(big):
        d = cases.laminar_case(nx=grid[0], ny=grid[1], nz=grid[2], lx=5.0, ly=3.0, lz=5.0)
        d.U[4, 4, 4] = big
        d.V[8, 3, 9] = -big
        d.W[3, 6, 10] = big
        return d

    inner = (slice(1, -1), slice(1, -1), slice(1, -1))
    ref = oracle.oracle_for(state(1.7e308)).smagorinsky()[inner]
    assert np.isinf(ref).sum() > 10 and np.isnan(ref).any() and np.isfinite(ref).sum() > 500
    for prec, big in ((FP64, 1.7e308), (MIXED, 3e38)):
        s = cases.solver_for(state(big), precision=prec, les_model=1)
        nut = s.compute_eddy_viscosity()[inner]
        assert np.array_equal(np.isinf(nut), np.isinf(ref)) and np.array_equal(np.isnan(nut), np.isnan(ref))
        ok = np.isfinite(ref)
        assert np.abs(nut[ok] - ref[ok]).max() <= (1e-14 if prec == FP64 else 1e-5) * np.abs(ref[ok]).max()
        s.close()


def test_les_steps_match_oracle(gpu):
    c = noisy(40, 13, 18, seed=22, amp=2e-3, cfl=-2e-3)
    s = cases.solver_for(c, les_model=1)
    o = oracle.oracle_for(c)
    o.set_les(1)
    for _ in range(4):
        s.time_step()
        o.step()
    U, V, W, _, _ = s.download_state()
    Ur, Vr, Wr, _, _ = o.state()
    assert rel(U, Ur) < 1e-10 and rel(V, Vr) < 1e-10 and rel(W, Wr) < 1e-10
    s.close()


def test_statistics_match_oracle(gpu):
    c = noisy(60, 17, 15, seed=23, amp=1e-3, cfl=-2e-3)
    s = cases.solver_for(c)
    o = oracle.oracle_for(c)
    for _ in range(2):
        s.time_step()
        o.step()
    a, b = s.compute_statistics(), o.statistics()
    for k in ("Umean", "Vmean", "Wmean", "U2mean", "V2mean", "W2mean", "UVmean", "Pmean", "P2mean", "Cf",
              "dUdy_wall"):
        assert rel(a[k], b[k]) < 1e-10, k
    for k in ("theta_inlet", "delta99_inlet", "Retheta_inlet"):
        assert a[k] == pytest.approx(b[k], rel=1e-10)
    s.close()


def test_law_of_the_wall_matches_oracle(gpu):
    c = cases.turbulent_case(nx=64, ny=49, nz=18, lx=10.0, ly=3.0, lz=2.0)
    s = cases.solver_for(c)
    o = oracle.oracle_for(c)
    guess = (0.5 * 0.027 * (c.x / c.nu) ** (-1.0 / 7.0)) ** 0.5  # utau_ref, initialization.f90:740
    u1, it1 = s.law_of_the_wall(guess)
    u2, it2 = o.law_of_the_wall(guess)
    assert it1 == it2 and it1 < 30
    assert np.abs(u1 - u2).max() <= 1e-12 * np.abs(u2).max()
    # the solution satisfies the log law at y = yg(3)
    yg = cases.centres_ghost(c.y)
    Um = c.U[1:-1, 2, 1:-1].mean(axis=1)
    f = u1[1:-1] / 0.38 * np.log(yg[2] * u1[1:-1] / c.nu) + 5.2 * u1[1:-1] - Um
    assert np.abs(f).max() < 1e-8
    s.close()


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_laminar_cfg1_skin_friction_blasius(gpu, precision):
    """Config 1: 200 RK3 steps at CFL 0.5; Cf(x) within 2% of 0.664/sqrt(Re_x)
    away from the inlet (3 points) and the outlet (5 points), as the
    reference's laminar_test/postprocess.py:164-170 compares it."""
    c = cases.laminar_case()
    s = cases.solver_for(c, precision=precision)
    s.advance(200)
    st = s.compute_statistics()
    rex = c.x / c.nu
    cf_bl = 0.664 / np.sqrt(rex)
    sl = slice(3, c.nx - 5)
    err = np.abs(st["Cf"][sl] - cf_bl[sl]) / cf_bl[sl]
    assert err.max() < 0.02, err.max()
    assert s.check_divergence() < (1e-12 if precision == FP64 else 1e-4)
    s.close()
