"""FP32 tile passes over grids in HBM, at the edges of their tiles (80 or 88
written rows, 14 lane columns of 8 cells): the launch-per-half-sweep kernels'
iterates, in a single solve and in a batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import poisson_caustic_design_gb300 as pcd

    c = pcd.Context(0)
    yield c
    c.close()


def _problem(n, m):
    import torch

    import poisson_caustic_design_gb300 as pcd

    b = pcd.inputs.poisson_rhs(max(n, m), 4, "binary" if n % 16 else "gaussian", m=max(n, m))[:m, :n]
    b = b - b.mean()
    start = 1e-2 * np.add.outer(np.cos(np.arange(m) / 7.0), np.sin(np.arange(n) / 5.0))
    return torch.from_numpy(np.ascontiguousarray(b)).cuda(), torch.from_numpy(start).cuda()


def _agree(x, ref):
    """FP32 rounding of the corrections, the other schedules' tolerance."""
    return bool((x - ref).abs().max() < 1e-5 * ref.abs().max())


@pytest.mark.parametrize("n", [8, 16, 112, 120, 128, 232])
@pytest.mark.parametrize("m", [1, 2, 15, 80, 81, 89, 161])
@pytest.mark.parametrize("check_every,sweeps", [(4, 1), (4, 43), (2, 37)])
def test_tile_edges(ctx, n, m, check_every, sweeps):
    import poisson_caustic_design_gb300 as pcd

    b, start = _problem(n, m)
    out = {}
    for sched in (1, 6):
        phi = start.clone()
        st = ctx.solve_device(b, phi, pcd.SolveOptions(
            stop=pcd.STOP_REL_RESIDUAL, tol=0.0, max_iterations=sweeps, precision=pcd.PREC_MIXED, omega=1.8,
            warm_start=1, schedule=sched, check_every=check_every if sched == 6 else 0, refine_every=16))
        assert st["sweeps"] == sweeps and st["schedule_used"] == sched
        out[sched] = phi
    assert _agree(out[6], out[1])


@pytest.mark.parametrize("zero_start", [False, True])
@pytest.mark.parametrize("narrow", [False, True])
def test_batch_tile_edges(ctx, zero_start, narrow):
    """Grids of unlike sizes in one batch, up to the sweep cap in the middle of
    a pass, are the single solves."""
    import torch

    import poisson_caustic_design_gb300 as pcd

    sizes = [(80, 112), (81, 120), (2, 16), (161, 232), (96, 128), (300, 1016)] + [(33, 8)] * narrow
    probs = [_problem(n, m) for m, n in sizes]
    o = dict(stop=pcd.STOP_REL_RESIDUAL, tol=1e-14, max_iterations=43, precision=pcd.PREC_MIXED, omega=1.8,
             refine_every=16)
    phis = [torch.full_like(s, 7.0) if zero_start else s.clone() for _, s in probs]
    stats, _ = pcd.solver.batch_solve(ctx, [b for b, _ in probs], phis,
                                      pcd.SolveOptions(warm_start=0 if zero_start else 1, **o))
    for (b, s), phi, st in zip(probs, phis, stats):
        assert st["sweeps"] == 43
        ref = torch.zeros_like(s) if zero_start else s.clone()
        ctx.solve_device(b, ref, pcd.SolveOptions(schedule=1, warm_start=1, **o))
        assert _agree(phi, ref)


@pytest.mark.parametrize("n,m", [(2048, 1500), (1600, 900), (1024, 704), (120, 89)])
@pytest.mark.parametrize("sweeps,refine_every", [(43, 41), (96, 32)])
def test_passes_without_a_barrier(ctx, n, m, sweeps, refine_every):
    """Launches of many passes, whose tiles wait only for their neighbours'
    last pass: more tiles than SMs (361, 180) and fewer (81, 4)."""
    import poisson_caustic_design_gb300 as pcd

    b, start = _problem(n, m)
    out = {}
    for sched in (1, 6):
        phi = start.clone()
        st = ctx.solve_device(b, phi, pcd.SolveOptions(
            stop=pcd.STOP_REL_RESIDUAL, tol=0.0, max_iterations=sweeps, precision=pcd.PREC_MIXED, omega=-1.0,
            warm_start=1, schedule=sched, refine_every=refine_every))
        assert st["sweeps"] == sweeps and st["schedule_used"] == sched
        out[sched] = phi
    assert _agree(out[6], out[1])


def test_tile_wait_runs_out():
    """With the first tile's passes never reported its neighbours' waits run
    out: the solve returns PCD_TIMEOUT and the context solves normally
    afterwards."""
    import poisson_caustic_design_gb300 as pcd

    c = pcd.Context(0)
    b, start = _problem(512, 512)
    o = pcd.SolveOptions(stop=pcd.STOP_REL_RESIDUAL, tol=1e-6, precision=pcd.PREC_MIXED, omega=-1.0, schedule=6)
    L = pcd.solver._lib.load()
    assert L.pcd_ctx_set_wait_limit(c.handle, 2000, 1) == 0
    with pytest.raises(pcd.PCDError) as err:
        c.solve_device(b, start.clone(), o)
    assert err.value.status == 4
    assert L.pcd_ctx_set_wait_limit(c.handle, 0, 0) == 0
    assert c.solve_device(b, start.clone(), o)["converged"]
    c.close()


# wider than the chip's registers hold, not a whole number of lane columns or of
# 16-byte rows: the last tile column in a whole and in a partial lane column, one
# cell to seven in it
RAGGED = [(1801, 1201, 1801), (1802, 1203, 1804), (1998, 1700, 2000), (2047, 1900, 2048), (1912, 1207, 1913),
          (4103, 600, 4104)]


def _auto(ctx, n, m, ld, sched, **kw):
    import torch

    import poisson_caustic_design_gb300 as pcd

    b0, start = _problem(n, m)
    b = torch.zeros((m, ld), dtype=torch.float64, device="cuda")[:, :n]
    phi = torch.zeros((m, ld), dtype=torch.float64, device="cuda")[:, :n]
    b.copy_(b0)
    phi.copy_(start)
    st = ctx.solve_device(b, phi, pcd.SolveOptions(precision=pcd.PREC_MIXED, omega=-1.0, schedule=sched, **kw))
    return st, phi


@pytest.mark.parametrize("n,m,ld", RAGGED)
@pytest.mark.parametrize("sweeps", [3, 75])
def test_ragged_grids_match_launch_schedule(ctx, n, m, ld, sweeps):
    ref = _auto(ctx, n, m, ld, 1, stop=1, tol=0.0, max_iterations=sweeps, refine_every=32)
    got = _auto(ctx, n, m, ld, 0, stop=1, tol=0.0, max_iterations=sweeps, refine_every=32)
    assert got[0]["sweeps"] == ref[0]["sweeps"] == sweeps
    assert _agree(got[1], ref[1])


@pytest.mark.parametrize("n,m,ld", RAGGED[:4])
@pytest.mark.parametrize("stop,tol,check_every", [(0, 2e-2, 0), (0, 2e-2, 3), (1, 0.3, 0)])
def test_ragged_grids_keep_their_stop_tests(ctx, n, m, ld, stop, tol, check_every):
    """AUTO's sweeps end where those of the schedule would that takes the grid
    otherwise: stream passes, or stripes."""
    ref = _auto(ctx, n, m, ld, 2, stop=stop, tol=tol, max_iterations=20000, check_every=check_every)
    assert ref[0]["schedule_used"] in (4, 5) and ref[0]["converged"]
    got = _auto(ctx, n, m, ld, 0, stop=stop, tol=tol, max_iterations=20000, check_every=check_every)
    assert got[0]["converged"] and got[0]["schedule_used"] == ref[0]["schedule_used"]
    assert got[0]["sweeps"] == ref[0]["sweeps"]
    assert _agree(got[1] - got[1].mean(), ref[1] - ref[1].mean())
