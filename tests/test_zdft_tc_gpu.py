"""The mixed form's z transforms on the tensor cores (TF32 products with a
three-term split; mma.sync and tcgen05 with tensor-memory accumulators):
against the FP32 direct sums and against the FP64 path, for odd and even z
lengths of every served order (M/2+1 rounded up to 16: 32, 48, 64, 80, 96)."""
import numpy as np
import pytest

from blgpu import cases, FP64, MIXED

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def noisy(nz, seed):
    c = cases.laminar_case(nx=34, ny=17, nz=nz, lx=10.0, ly=5.0, lz=4.0)
    rng = np.random.default_rng(seed)
    c.U = np.asfortranarray(c.U + 0.05 * rng.standard_normal(c.U.shape))
    c.V = np.asfortranarray(c.V + 0.05 * rng.standard_normal(c.V.shape))
    c.W = np.asfortranarray(c.W + 0.05 * rng.standard_normal(c.W.shape))
    c.cfl = -0.01
    return c


@pytest.mark.parametrize("form", [2, 3])
@pytest.mark.parametrize("nz", [64, 65, 96, 97, 127, 159, 193, 194])
def test_tensor_core_z_transform_matches_direct_and_fp64(gpu, nz, form):
    c = noisy(nz, nz)
    out = {}
    for name, prec, zdft in (("tc", MIXED, form), ("direct", MIXED, 1), ("fp64", FP64, 0)):
        s = cases.solver_for(c, precision=prec)
        if prec == MIXED:
            s.set_tiles(zdft=zdft)
        # boundary pass before (compatible Neumann problem) and after (ghost
        # cells the divergence check reads), as in a substep
        s.apply_boundary_conditions(1)
        s.compute_projection_step(1)
        s.apply_boundary_conditions(1)
        out[name] = (s.download_state()[:3], s.rhs_p(), s.check_divergence())
        s.close()
    (Ut, Vt, Wt), pt, dt = out["tc"]
    (Ud, Vd, Wd), pd, dd = out["direct"]
    (U6, V6, W6), p6, d6 = out["fp64"]
    # FP32 pressure against FP64 on a noisy field (both z-transform forms
    # alike), then the two forms against each other
    assert rel(pt, p6) < 3e-5 and rel(pd, p6) < 3e-5, (rel(pt, p6), rel(pd, p6))
    assert rel(pt, pd) < 1e-5
    for a, b in ((Ut, U6), (Vt, V6), (Wt, W6)):
        assert rel(a, b) < 1e-5
    assert dt < 1e-3 and dt <= 10 * dd + 1e-6


@pytest.mark.parametrize("form", [0, 2, 3])
def test_tensor_core_path_steps_close_to_fp64(gpu, form):
    c = cases.turbulent_case(nx=66, ny=33, nz=193, lx=8.0, ly=2.0, lz=8.0, seed=9, cfl=-0.01)
    a = cases.solver_for(c, precision=MIXED)
    assert a.tiles()["zdft"] == 0
    a.set_tiles(zdft=form)
    b = cases.solver_for(c, precision=FP64)
    a.advance(10)
    b.advance(10)
    A, B = a.download_state()[:3], b.download_state()[:3]
    for x, y in zip(A, B):
        assert rel(x, y) < 1e-5


@pytest.mark.parametrize("nx,nz", [(34, 194), (71, 195), (66, 225), (35, 255), (67, 256), (130, 257), (34, 258),
                                   (36, 259), (34, 402)])
def test_long_z_transform_products_close_to_fp64(gpu, nx, nz):
    """z lengths beyond the tensor-core kernels (M/2+1 = 97 .. 201, odd and
    even M): slabs of 16 table rows (97 and 113 leave 15 padded, 128 none),
    row tiles of 128 (128 and 129 rows), columns that end inside a 64-column
    tile (N = 32, 69) and inside a group of four (69, 33, 65)."""
    c = cases.laminar_case(nx=nx, ny=9, nz=nz, lx=10.0, ly=5.0, lz=8.0)
    rng = np.random.default_rng(nz)
    for q in "UVW":
        a = getattr(c, q)
        setattr(c, q, np.asfortranarray(a + 0.05 * rng.standard_normal(a.shape)))
    c.cfl = -0.01
    out = []
    for prec in (MIXED, FP64):
        s = cases.solver_for(c, precision=prec)
        s.apply_boundary_conditions(1)
        s.compute_projection_step(1)
        s.apply_boundary_conditions(1)
        out.append((s.download_state()[:3], s.rhs_p()))
        s.close()
    (A, pa), (B, pb) = out
    assert rel(pa, pb) < 3e-5  # the direct sums' bar above
    for a, b in zip(A, B):
        assert rel(a, b) < 1e-5


@pytest.mark.parametrize("nz", [194, 258, 402, 455])
def test_long_z_transform_products_match_direct_sums(gpu, nz):
    """zdft 1 selects the direct sums beyond the tensor-core lengths as well,
    to M = 453 (nz = 455), with 4 or 8 wavenumbers per warp: the same FP32
    transform as the products, for odd M to the bit (the same terms in the same
    order), for even M to the rounding of sums of M/2 terms (the term M/2 is
    added first in one form and last in the other)."""
    c = noisy(nz, nz)
    out = []
    for tiles in ({}, {"zdft": 1}, {"zdft": 1, "dftz_rk": 4}, {"zdft": 1, "dftz_rk": 8}):
        s = cases.solver_for(c, precision=MIXED)
        s.set_tiles(**tiles)
        s.apply_boundary_conditions(1)
        s.compute_projection_step(1)
        out.append(s.rhs_p())
        s.close()
    assert rel(out[0], out[1]) < 1e-5
    assert np.array_equal(out[0], out[1]) == (nz % 2 == 1)
    assert np.array_equal(out[1], out[2]) and np.array_equal(out[1], out[3])


@pytest.mark.parametrize("nx,nz", [(34, 456), (21, 514), (34, 641), (34, 768), (40, 769)])
def test_longest_z_transform_products_match_oracle(gpu, nx, nz):
    """Beyond the direct sums' shared memory (M > 453) up to the products'
    limit M = 767, the largest columns (M/2+1 = 384) and row tiles of 128 that
    end full and not (257 and 321 rows, 384): the projection against the FP64
    oracle at the bars of the shorter lengths."""
    import oracle
    c = cases.laminar_case(nx=nx, ny=6, nz=nz, lx=10.0, ly=5.0, lz=16.0)
    rng = np.random.default_rng(nz)
    for q in "UVW":
        a = getattr(c, q)
        setattr(c, q, np.asfortranarray(a + 0.05 * rng.standard_normal(a.shape)))
    o = oracle.oracle_for(c)
    s = cases.solver_for(c, precision=MIXED)
    o.set_dt(0.01)
    s.set_dt(0.01)
    o.apply_bc(1)
    s.apply_boundary_conditions(1)
    o.projection(1)
    s.compute_projection_step(1)
    assert rel(s.rhs_p()[:, :, :-1], o.rhs_p()[:, :, :-1]) < 3e-5
    for a, b in zip(s.download_state()[:3], o.state()[:3]):
        assert rel(a, b) < 1e-5
    s.close()


@pytest.mark.parametrize("prec,nz", [(MIXED, 770), (FP64, 456)])
def test_z_lengths_past_shared_memory_are_refused(gpu, prec, nz):
    """No z transform holds M = 768 columns in the mixed form, or 454 in FP64:
    projections and steps say so instead of going on without the transform, and
    neither the context nor the next one is left with an error."""
    from blgpu import BlgpuError, Ensemble
    c = cases.laminar_case(nx=10, ny=6, nz=nz, lx=10.0, ly=5.0, lz=16.0)
    s = cases.solver_for(c, precision=prec)
    s.set_dt(0.01)
    s.apply_boundary_conditions(1)
    ens = Ensemble([s])
    for call in (lambda: s.compute_projection_step(1), s.time_step, lambda: s.advance(1), lambda: s.phase_times(1),
                 lambda: ens.advance(1)):
        with pytest.raises(BlgpuError, match="z transforms hold"):
            call()
    ens.close()
    s.sync()
    assert np.isfinite(s.compute_rhs(c.U, c.V, c.W)[0]).all()
    s.close()
    cases.solver_for(c, precision=prec).close()


@pytest.mark.parametrize("nx,ny", [(5, 4), (64, 5), (65, 6), (66, 9), (128, 8), (129, 17), (200, 10)])
def test_box_scale_pressure_tiles(gpu, nx, ny):
    """The mixed form's FP64 box-scale pressure and its differences at the
    edges of their tiles: 63 columns (N = 62, 63, 64, 126, 127), 4 rows
    (ny-1 = 3, 4, 5, 8, 7, 16, 9) and fewer modes than 128 (N = 3): the
    projected velocities against FP64."""
    c = cases.laminar_case(nx=nx, ny=ny, nz=12, lx=10.0, ly=5.0, lz=4.0)
    rng = np.random.default_rng(nx)
    for q in "UVW":
        a = getattr(c, q)
        setattr(c, q, np.asfortranarray(a + 0.05 * rng.standard_normal(a.shape)))
    c.cfl = -0.01
    out = []
    for prec in (MIXED, FP64):
        s = cases.solver_for(c, precision=prec)
        s.apply_boundary_conditions(1)
        s.compute_projection_step(1)
        s.apply_boundary_conditions(1)
        out.append((s.download_state()[:3], s.rhs_p()))
        s.close()
    (A, pa), (B, pb) = out
    assert rel(pa, pb) < 3e-5
    for a, b in zip(A, B):
        assert rel(a, b) < 1e-5
