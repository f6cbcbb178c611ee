"""The FP64 block kernel at the edges of its layouts: odd widths (a pair's
second column outside the grid), blocks as tall as their halo, one block row or
column, 1, 2 and 4 sweeps per exchange."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import poisson_caustic_design_gb300 as pcd

    c = pcd.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n,m", [(64, 64), (65, 71), (57, 300), (56, 64), (113, 37), (255, 257), (512, 130), (767, 500)])
@pytest.mark.parametrize("k", [0, 1, 2, 4])
@pytest.mark.parametrize("sweeps", [1, 23])
def test_blocks64_match_launch_schedule(ctx, n, m, k, sweeps):
    """The same iterate after the same sweeps, to the rounding of the two
    summation orders (the block schedule's tolerance)."""
    import poisson_caustic_design_gb300 as pcd

    b = pcd.inputs.poisson_rhs(n, 4, "binary" if m % 2 else "gaussian", m=m)
    start = 1e-2 * np.add.outer(np.cos(np.arange(m) / 7.0), np.sin(np.arange(n) / 5.0))
    out = {}
    for sched in (pcd.SCHED_LAUNCHES, pcd.SCHED_BLOCKS):
        phi = start.copy()
        st = ctx.solve(b, phi, pcd.SolveOptions(stop=pcd.STOP_REL_RESIDUAL, tol=0.0, max_iterations=sweeps,
                                                schedule=sched, omega=1.9,
                                                block_sweeps=k if sched == pcd.SCHED_BLOCKS else 0))
        assert st["sweeps"] == sweeps
        out[sched] = phi
    a, c = out[pcd.SCHED_LAUNCHES], out[pcd.SCHED_BLOCKS]
    assert np.abs(a - c).max() <= 1e-11 * np.abs(a).max()


@pytest.mark.parametrize("n,m", [(64, 64), (255, 130)])
def test_blocks64_max_update_is_the_last_sweeps(ctx, n, m):
    """The max-update stop tests the sweep before each test: the reported
    value is the largest change of that sweep."""
    import poisson_caustic_design_gb300 as pcd

    b = pcd.inputs.poisson_rhs(n, 6, "gaussian", m=m)
    its = []
    for sweeps in (31, 32):
        phi = np.zeros_like(b)
        st = ctx.solve(b, phi, pcd.SolveOptions(stop=pcd.STOP_MAX_UPDATE, tol=0.0, max_iterations=sweeps, omega=1.9,
                                                schedule=pcd.SCHED_BLOCKS))
        its.append(phi)
    assert st["sweeps"] == 32
    assert abs(st["last_max_update"] - np.abs(its[1] - its[0]).max()) <= 1e-11 * np.abs(b).max() * n
