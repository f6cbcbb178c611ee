"""Fields beyond 32-bit byte offsets: rows further apart than the FP64 refresh
takes, and more than 4 GB in a field."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def ctx():
    import poisson_caustic_design_gb300 as pcd

    c = pcd.Context(0)
    yield c
    c.close()


def _grid(m, n, ld):
    import torch

    return torch.empty((m - 1) * ld + n, dtype=torch.float64, device="cuda").as_strided((m, n), (ld, 1))


@pytest.mark.parametrize("stop", [0, 1])
def test_rows_too_far_apart_for_the_refresh(ctx, stop):
    """ld of 2^26 and more: AUTO falls back, and its solution is the compact grid's."""
    import torch

    import poisson_caustic_design_gb300 as pcd

    m, n = 20, 40
    o = pcd.SolveOptions(stop=stop, tol=1e-10, precision=pcd.PREC_MIXED, omega=-1.0, warm_start=0,
                         max_iterations=20000)
    rhs = torch.from_numpy(pcd.inputs.poisson_rhs(n, 4, "gaussian", m=m)).cuda()
    ref = torch.zeros_like(rhs)
    assert ctx.solve_device(rhs, ref, o)["converged"]
    b, phi = _grid(m, n, (1 << 26) + 4), _grid(m, n, (1 << 26) + 4)
    b.copy_(rhs)
    st = ctx.solve_device(b, phi, o)
    assert st["converged"] and st["schedule_used"] != pcd.SCHED_TILES
    a, c = phi - phi.mean(), ref - ref.mean()
    assert (a - c).abs().max() < 1e-7 * c.abs().max()


def test_field_beyond_4_gb(ctx):
    """131072 x 4100 cells: a strip of the refresh is cut where its byte offsets would
    leave 32 bits (4092 rows).  The launch schedule's iterate after two sweeps, each with its refresh."""
    import torch

    import poisson_caustic_design_gb300 as pcd

    m, n = 4100, 131072
    x = torch.arange(n, dtype=torch.float64, device="cuda")
    y = torch.arange(m, dtype=torch.float64, device="cuda")
    b, start, phi = _grid(m, n, n), _grid(m, n, n), _grid(m, n, n)
    torch.outer(torch.cos(y / 11.0), torch.sin(x / 13.0), out=b)
    torch.outer(torch.sin(y / 5.0), torch.cos(x / 7.0), out=start)
    o = dict(stop=pcd.STOP_REL_RESIDUAL, tol=0.0, max_iterations=2, refine_every=1, precision=pcd.PREC_MIXED,
             omega=1.8, warm_start=1)
    phi.copy_(start)
    assert ctx.solve_device(b, phi, pcd.SolveOptions(schedule=pcd.SCHED_AUTO, **o))["schedule_used"] == pcd.SCHED_TILES
    ctx.solve_device(b, start, pcd.SolveOptions(schedule=pcd.SCHED_LAUNCHES, **o))
    start_max = start.abs().max()
    assert (phi - start).abs_().max() < 1e-5 * start_max


def test_grid_beyond_memory_is_refused_and_the_context_goes_on(ctx):
    """A grid whose workspace cannot be had (429 GB of its smallest buffer alone) is
    an error, and the next solve works on buffers of its own again."""
    import ctypes

    import torch

    import poisson_caustic_design_gb300 as pcd

    b = torch.from_numpy(pcd.inputs.poisson_rhs(64, 4, "gaussian")).cuda()
    o = pcd.SolveOptions(stop=1, tol=1e-6, precision=pcd.PREC_MIXED, omega=-1.0, warm_start=0)
    out = []
    for _ in range(2):
        phi = torch.zeros_like(b)
        assert ctx.solve_device(b, phi, o)["converged"]
        out.append(phi)
        st = pcd._lib.SolveStats()
        c = o.to_c()
        rc = pcd._lib.load().pcd_poisson_solve_device(ctx.handle, b.data_ptr(), phi.data_ptr(), 16, 200, 2**31 - 1,
                                                      ctypes.byref(c), ctypes.byref(st), None)
        assert rc == pcd._lib.PCD_DEVICE_ERROR
    assert torch.equal(*out)
