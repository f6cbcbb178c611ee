"""Narrow grids on the schedules made for wide ones: one sweep a launch on the
register-resident cluster form, and stream passes whose block has more threads than
the row has cells."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import poisson_caustic_design_gb300 as pcd

    c = pcd.Context(0)
    yield c
    c.close()


def _same(ctx, n, m, ld, schedule, **kw):
    import torch

    import poisson_caustic_design_gb300 as pcd

    rhs = pcd.inputs.poisson_rhs(max(n, m), 4, "gaussian", m=max(n, m))[:m, :n]
    rhs = rhs - rhs.mean()
    start = 1e-2 * np.add.outer(np.cos(np.arange(m) / 7.0), np.sin(np.arange(n) / 5.0))
    out = []
    for sched in (pcd.SCHED_LAUNCHES, schedule):
        b = torch.zeros((m, ld), dtype=torch.float64, device="cuda")[:, :n]
        phi = torch.zeros((m, ld), dtype=torch.float64, device="cuda")[:, :n]
        b.copy_(torch.from_numpy(rhs))
        phi.copy_(torch.from_numpy(start))
        st = ctx.solve_device(b, phi, pcd.SolveOptions(tol=0.0, omega=1.8, warm_start=1, schedule=sched,
                                                       precision=pcd.PREC_MIXED, **kw))
        assert st["sweeps"] == kw["max_iterations"] and st["schedule_used"] == sched
        out.append(phi)
    assert (out[0] - out[1]).abs().max() < 1e-5 * out[0].abs().max()


@pytest.mark.parametrize("n,m", [(8, 33), (8, 188), (8, 252), (320, 48), (384, 768)])
@pytest.mark.parametrize("refine_every,sweeps", [(1, 1), (1, 300), (2, 37)])
def test_cluster_launches_of_few_sweeps(ctx, n, m, refine_every, sweeps):
    """A launch's first halo stores come a few microseconds after its start."""
    _same(ctx, n, m, n, 3, stop=1, refine_every=refine_every, max_iterations=sweeps)


@pytest.mark.parametrize("n,m,ld", [(1, 40, 4), (5, 40, 8), (17, 3, 20), (24, 33, 24), (130, 20, 132), (2050, 9, 2052)])
@pytest.mark.parametrize("stop", [0, 1])
def test_stream_passes_on_narrow_rows(ctx, n, m, ld, stop):
    _same(ctx, n, m, ld, 5, stop=stop, refine_every=16, max_iterations=37)
