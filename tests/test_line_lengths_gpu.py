"""The Poisson solve and the step over every compiled line length, in x and in y, with column
heights around the groups of eight rows that the tridiagonal sweeps work in."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [16, 18, 24, 32, 36, 48, 54, 72, 96, 108, 128, 144, 162, 216, 288, 324, 432, 486, 576, 648, 864, 972]


def rhs_and_reference(O, nx, ny, nz, nparts=0):
    g = O.Grid(nx, ny, nz, stretch=1.6)
    r = np.random.default_rng(nx * 1000 + ny + nz).standard_normal((nz, ny, nx))
    wgt = g.dzf_global[1:-1]
    r -= (r.mean(axis=(1, 2)) * wgt).sum() / wgt.sum()
    var = np.zeros(g.shape)
    var[1:-1, 1:-1, 1:-1] = r
    O.PPE(nx, ny, nz, g.g.dx, g.g.dy, g.dzf_global, nparts=nparts).execute(var)
    p = var[1:-1, 1:-1, 1:-1]
    return g, r, p - p.mean()


def solve(plb, g, r, precision, nparts=0):
    import torch
    nz, ny, nx = r.shape
    s = plb.DevicePoissonSolver(nx, ny, nz, g.g.dx, g.g.dy, g.dzf_global, nparts=nparts, precision=precision)
    x = torch.tensor(r, dtype=torch.float64 if precision == plb.PL_FP64 else torch.float32, device="cuda")
    s.solve(x)
    torch.cuda.synchronize()
    p = x.cpu().numpy().astype(np.float64)
    return p - p.mean()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("n", LENGTHS)
def test_solve_by_line_length(gpu, oracle_mod, n, precision, tol):
    """x of length n over y of the next length and the other way round (ny/2 not a multiple of the
    lines a group holds; odd column counts), at a height of ten rows.  Tolerances as for the
    other lengths: the FP64 bar, and FP32 transforms."""
    plb, O = gpu, oracle_mod
    other = LENGTHS[(LENGTHS.index(n) + 1) % 6]
    for nx, ny in ((n, other), (other, n)):
        g, r, ref = rhs_and_reference(O, nx, ny, 10)
        got = solve(plb, g, r, plb.PL_FP64 if precision == "fp64" else plb.PL_MIXED)
        assert np.abs(got - ref).max() < tol * np.abs(ref).max(), (nx, ny)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("nz", [2, 6, 14, 22, 150, 250, 254, 258, 274, 306])
def test_solve_by_column_height(gpu, oracle_mod, nz, precision, tol):
    """Heights that the groups of eight rows do not divide, up to and beyond the 256 rows that
    tensor memory holds; 162 columns a row, so the last CTA is partly empty."""
    plb, O = gpu, oracle_mod
    g, r, ref = rhs_and_reference(O, 162, 16, nz)
    got = solve(plb, g, r, plb.PL_FP64 if precision == "fp64" else plb.PL_MIXED)
    assert np.abs(got - ref).max() < tol * np.abs(ref).max()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("nz,nparts", [(64, 4), (96, 6), (120, 5), (128, 8), (192, 3)])
def test_pdd_by_partition_size(gpu, oracle_mod, nz, nparts, precision, tol):
    """Partitions of 8, 16, 24 and 64 rows: loads of 8 and of 16 rows."""
    plb, O = gpu, oracle_mod
    g, r, ref = rhs_and_reference(O, 54, 18, nz, nparts)
    got = solve(plb, g, r, plb.PL_FP64 if precision == "fp64" else plb.PL_MIXED, nparts)
    assert np.abs(got - ref).max() < tol * np.abs(ref).max()


def test_pdd_on_an_array_larger_than_l2(gpu, oracle_mod):
    """151 MB in partitions of 24 rows: batches of 8 rows whose successors are requested into L2."""
    plb, O = gpu, oracle_mod
    g, r, ref = rhs_and_reference(O, 512, 384, 96, 4)
    got = solve(plb, g, r, plb.PL_FP64, 4)
    assert np.abs(got - ref).max() < 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("nx,ny,nz,nparts", [(162, 64, 48, 3), (128, 72, 64, 4), (16, 648, 48, 3), (216, 96, 384, 8)])
def test_pdd_two_columns_per_thread(gpu, oracle_mod, nx, ny, nz, nparts, precision, tol):
    """At least 148 CTAs of mirrored column pairs: a ragged last CTA, the rows without a mirror (0 and
    ny / 2), exactly 148, and partitions whose pairs take 384 of the 512 cells."""
    plb, O = gpu, oracle_mod
    g, r, ref = rhs_and_reference(O, nx, ny, nz, nparts)
    got = solve(plb, g, r, plb.PL_FP64 if precision == "fp64" else plb.PL_MIXED, nparts)
    assert np.abs(got - ref).max() < tol * np.abs(ref).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,nz", [(16, 6, 4), (54, 18, 14), (96, 24, 22), (162, 16, 10), (324, 8, 6)])
def test_step_matches_phases(gpu, precision, nx, ny, nz):
    """calcRHS inside the forward x transform (several lines per group at short lengths, the
    last group of a plane partly filled) against calcRHS as its own kernel: FP64 bit for bit;
    mixed to 1e-11, the plane sums being added in another order."""
    plb = gpu
    cfg = plb.ChannelConfig(nx=nx, ny=ny, nz=nz, stretch_ratio=1.5, re_tau=180.0,
                            precision=plb.PL_FP64 if precision == "fp64" else plb.PL_MIXED)
    a, b = plb.Channel(cfg), plb.Channel(cfg)
    for ch in (a, b):
        ch.init_flow(5, 0.1)
    for _ in range(4):
        a.step(1)
        for ph in ("rk", "calc_rhs", "poisson", "correct_force"):
            b.phase(ph)
    for x, y in zip(a.get_fields()[:3], b.get_fields()[:3]):
        if precision == "fp64":
            assert np.array_equal(x, y)
        else:
            assert np.abs(x - y).max() < 1e-11 * np.abs(y).max()
    a.close()
    b.close()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("nz", [1016, 1022, 1024, 1026, 1032])
def test_solve_by_tall_column(gpu, oracle_mod, nz, precision, tol):
    """Around the 1,024 rows up to which the sweep uses tensor memory: above them its values are
    swept through device memory alone."""
    plb, O = gpu, oracle_mod
    g, r, ref = rhs_and_reference(O, 16, 18, nz)
    got = solve(plb, g, r, plb.PL_FP64 if precision == "fp64" else plb.PL_MIXED)
    assert np.abs(got - ref).max() < tol * np.abs(ref).max()


@pytest.mark.parametrize("nx,ny,nz,nparts,precision", [
    (512, 384, 192, 8, "mixed"),                                 # batches of 8 rows, one column a thread
    (192, 162, 576, 4, "fp64"), (288, 216, 576, 4, "mixed"),     # 16 rows, one column: 144 rows a partition
    (512, 384, 96, 3, "fp64"), (512, 384, 192, 4, "mixed")])     # 16 rows, two columns
def test_pdd_variants_on_arrays_larger_than_l2(gpu, oracle_mod, nx, ny, nz, nparts, precision):
    """143 to 151 MB: the variants of the partition sweep that request the next batch of rows into L2."""
    plb, O = gpu, oracle_mod
    g, r, ref = rhs_and_reference(O, nx, ny, nz, nparts)
    got = solve(plb, g, r, plb.PL_FP64 if precision == "fp64" else plb.PL_MIXED, nparts)
    assert np.abs(got - ref).max() < (1e-12 if precision == "fp64" else 1e-5) * np.abs(ref).max()


@pytest.mark.parametrize("nparts", [0, 3])
@pytest.mark.parametrize("n", LENGTHS)
def test_host_solve_by_line_length(gpu, oracle_mod, n, nparts):
    """init/execute/free_poisson_solver: the strided x transforms of every length on the ghosted
    host array, whose ghosts stay untouched.  The FP64 bar."""
    plb, O = gpu, oracle_mod
    ny, nz = LENGTHS[(LENGTHS.index(n) + 1) % 6], 12
    g, r, ref = rhs_and_reference(O, n, ny, nz, nparts)
    var = np.full((nz + 2, ny + 2, n + 2), 7.25)
    var[1:-1, 1:-1, 1:-1] = r
    with plb.PoissonSolver(n, ny, nz, g.g.dx, g.g.dy, g.dzf_global, nparts=nparts) as s:
        s.execute(var)
    got = var[1:-1, 1:-1, 1:-1].copy()
    var[1:-1, 1:-1, 1:-1] = 7.25
    assert np.all(var == 7.25)
    assert np.abs((got - got.mean()) - ref).max() < 1e-12 * np.abs(ref).max()
