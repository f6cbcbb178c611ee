"""FP32 sweeps on tiles that stay on the chip (AUTO's form for mixed solves on
grids that fit): the same iterates, sweep counts and stops as the schedules
whose stop tests they keep."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one tile (rows and columns), tile columns with a one-lane remainder, odd
# heights and widths, partial lane columns of 1 to 7 cells, the two row
# heights, 8 and 4 sweeps per exchange, the largest tiles
SHAPES = [(16, 16), (17, 19), (56, 64), (64, 48), (65, 33), (100, 36), (120, 129), (127, 301), (128, 128), (252, 188),
          (511, 64), (512, 33), (512, 512), (640, 480), (1000, 900), (1032, 1024), (1536, 1281)]


@pytest.fixture(scope="module")
def ctx():
    import poisson_caustic_design_gb300 as pcd

    c = pcd.Context(0)
    yield c
    c.close()


def _solve(ctx, b, phi0=None, ld=None, **kw):
    import torch

    import poisson_caustic_design_gb300 as pcd

    h, w = b.shape
    ld = ld or w
    bd = torch.zeros((h, ld), dtype=torch.float64, device="cuda")[:, :w]
    bd.copy_(torch.from_numpy(b))
    phi = torch.zeros((h, ld), dtype=torch.float64, device="cuda")[:, :w]
    if phi0 is not None:
        phi.copy_(torch.from_numpy(phi0))
    st = ctx.solve_device(bd, phi, pcd.SolveOptions(precision=pcd.PREC_MIXED, **kw))
    return st, phi.cpu().numpy()


@pytest.mark.parametrize("n,m", SHAPES)
@pytest.mark.parametrize("sweeps", [1, 37])
def test_resident_sweeps_match_launch_schedule(ctx, n, m, sweeps):
    """After the same number of sweeps the iterates agree to FP32 rounding
    (the tolerance of the other schedules' tests)."""
    import poisson_caustic_design_gb300 as pcd

    b = pcd.inputs.poisson_rhs(n, 5, "binary" if m % 2 else "gaussian", m=m)
    out = {}
    for sched in (1, 0):
        st, out[sched] = _solve(ctx, b, stop=1, tol=1e-14, max_iterations=sweeps, omega=1.9, schedule=sched)
        assert st["sweeps"] == sweeps
    assert st["schedule_used"] == 6
    assert np.abs(out[0] - out[1]).max() < 1e-5 * np.abs(out[1]).max()


@pytest.mark.parametrize("n,m,ld,tol", [(64, 64, 64, 1e-7), (200, 136, 204, 1e-5), (512, 300, 512, 1e-5),
                                        (1024, 700, 1024, 1e-4)])
@pytest.mark.parametrize("check_every", [0, 3])
def test_resident_max_update_stop_is_the_tile_passes(ctx, n, m, ld, tol, check_every):
    """The max-update stop is found after the fact and the chunk run again up
    to the sweep that passed: the same sweeps and the same bits as the passes
    that test after every pass, from a zero and from a given start."""
    import poisson_caustic_design_gb300 as pcd

    b = pcd.inputs.poisson_rhs(n, 6, "gaussian", m=m)
    start = 1e-2 * np.add.outer(np.cos(np.arange(m) / 7.0), np.sin(np.arange(n) / 5.0))
    for phi0 in (None, start):
        res = [_solve(ctx, b, phi0, ld, stop=0, tol=tol, omega=-1.0, schedule=s, check_every=check_every)
               for s in (0, 6)]
        assert res[0][0]["converged"] and res[1][0]["converged"]
        assert res[0][0]["sweeps"] == res[1][0]["sweeps"]
        assert res[0][0]["last_max_update"] == res[1][0]["last_max_update"]
        np.testing.assert_array_equal(res[0][1], res[1][1])


@pytest.mark.parametrize("n,m,other", [(64, 48, 3), (512, 512, 3), (252, 188, 3), (300, 260, 3), (768, 640, 6)])
def test_resident_residual_stop_matches(ctx, n, m, other):
    """The relative-residual stop keeps the cluster's estimate cycles (whole
    and partial lane columns) and the tile passes' chunks: the same sweeps,
    and the same solution, up to the constant that the Neumann problem leaves
    open, to a thousandth of the tolerance."""
    import poisson_caustic_design_gb300 as pcd

    b = pcd.inputs.poisson_rhs(n, 7, "binary", m=m)
    res = [_solve(ctx, b, stop=1, tol=1e-6, omega=-1.0, warm_start=0, schedule=s) for s in (0, other)]
    assert res[0][0]["converged"] and res[0][0]["schedule_used"] == 6 and res[1][0]["schedule_used"] == other
    assert res[0][0]["sweeps"] == res[1][0]["sweeps"]
    d = res[0][1] - res[1][1]
    assert np.abs(d - d.mean()).max() < 1e-9 * np.abs(res[1][1]).max()


def test_resident_wait_runs_out():
    """With the first tile's words withheld its neighbours' waits run out: the
    solve returns PCD_TIMEOUT and the context solves normally afterwards."""
    import poisson_caustic_design_gb300 as pcd

    c = pcd.Context(0)
    b = pcd.inputs.poisson_rhs(256, 3, "gaussian")
    L = pcd.solver._lib.load()
    assert L.pcd_ctx_set_wait_limit(c.handle, 2000, 1) == 0
    with pytest.raises(pcd.PCDError) as err:
        _solve(c, b, stop=1, tol=1e-6, omega=-1.0)
    assert err.value.status == 4
    assert L.pcd_ctx_set_wait_limit(c.handle, 0, 0) == 0
    st, _ = _solve(c, b, stop=1, tol=1e-6, omega=-1.0)
    assert st["converged"] and st["schedule_used"] == 6
    c.close()


@pytest.mark.parametrize("n,m,ld,schedule,used,form", [
    (512, 512, 512, 0, 6, 1), (512, 512, 512, 6, 6, 2), (252, 188, 252, 0, 6, 1), (2048, 1500, 2048, 0, 6, 2),
    (1801, 1201, 1801, 0, 4, 2), (2044, 1500, 2044, 0, 5, 2), (512, 512, 512, 3, 3, 0), (512, 512, 512, 1, 1, 0)])
def test_stats_tell_what_the_sweeps_ran_on(ctx, n, m, ld, schedule, used, form):
    """schedule_used names whose stop tests a solve keeps; sweep_form the kernel."""
    import poisson_caustic_design_gb300 as pcd

    b = pcd.inputs.poisson_rhs(max(n, m), 5, "gaussian", m=max(n, m))[:m, :n]
    st, _ = _solve(ctx, b, ld=ld, stop=1, tol=1e-14, max_iterations=8, omega=1.9, schedule=schedule)
    assert (st["schedule_used"], st["sweep_form"]) == (used, form)


# one grid for each instance of the kernel that a plan takes: sweeps per exchange, rows
# and lane columns of a lane group, whole and partial lane columns
@pytest.mark.parametrize("n,m", [(72, 16), (72, 17), (776, 2310), (792, 2436), (16, 144), (200, 2436), (456, 2401),
                                 (584, 2359), (17, 16), (65, 16), (65, 17), (17, 144), (193, 2436)])
def test_every_instance_matches_launch_schedule(ctx, n, m):
    import poisson_caustic_design_gb300 as pcd

    b = pcd.inputs.poisson_rhs(max(n, m), 5, "gaussian", m=max(n, m))[:m, :n]
    b = b - b.mean()
    out = {}
    for sched in (1, 0):
        st, out[sched] = _solve(ctx, b, stop=1, tol=1e-14, max_iterations=37, omega=1.9, schedule=sched)
        assert st["sweeps"] == 37
    assert st["sweep_form"] == 1
    assert np.abs(out[0] - out[1]).max() < 1e-5 * np.abs(out[1]).max()
