"""Batched tile passes whose waits between tiles run out (failure handling without a
GPU fault)."""
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(161, 232), (96, 128), (300, 1016), (64, 64)]  # several tiles, one, several, one


@pytest.fixture
def ctx():
    import poisson_caustic_design_gb300 as pcd

    c = pcd.Context(0)
    yield c
    c.close()


def _grids():
    import numpy as np
    import torch

    import poisson_caustic_design_gb300 as pcd

    bs = [torch.from_numpy(pcd.inputs.poisson_rhs(n, 4, "gaussian", m=m)).cuda() for m, n in SIZES]
    starts = [torch.from_numpy(1e-2 * np.add.outer(np.cos(np.arange(m) / 7.0), np.sin(np.arange(n) / 5.0))).cuda()
              for m, n in SIZES]
    return bs, starts


def _options(**kw):
    import poisson_caustic_design_gb300 as pcd

    return pcd.SolveOptions(stop=pcd.STOP_REL_RESIDUAL, tol=1e-6, precision=pcd.PREC_MIXED, omega=-1.0, **kw)


def test_batch_wait_runs_out(ctx):
    """With the first tile never reported done its neighbours' waits run out: the batch
    returns PCD_TIMEOUT, and the context solves the next one as any other does."""
    import torch

    import poisson_caustic_design_gb300 as pcd

    bs, starts = _grids()
    L = pcd._lib.load()
    assert L.pcd_ctx_set_wait_limit(ctx.handle, 2000, 1) == 0
    with pytest.raises(pcd.PCDError) as err:
        pcd.batch_solve(ctx, bs, [s.clone() for s in starts], _options(max_iterations=200))
    assert err.value.status == pcd._lib.PCD_TIMEOUT
    assert L.pcd_ctx_set_wait_limit(ctx.handle, 0, 0) == 0
    got, ref = [s.clone() for s in starts], [s.clone() for s in starts]
    stats, _ = pcd.batch_solve(ctx, bs, got, _options())
    assert all(st["converged"] for st in stats)
    other = pcd.Context(0)
    pcd.batch_solve(other, bs, ref, _options())
    other.close()
    assert all(torch.equal(a, b) for a, b in zip(got, ref))


def test_batch_stops_at_the_wait_that_ran_out(ctx):
    """The chunk that failed is the last one, and no grid's potential takes up what its
    tiles had left undone: with the failure in the first chunk each is its start."""
    import torch

    import poisson_caustic_design_gb300 as pcd

    bs, starts = _grids()
    phis = [s.clone() for s in starts]
    L = pcd._lib.load()
    assert L.pcd_ctx_set_wait_limit(ctx.handle, 2000, 1) == 0
    before = L.pcd_kernel_launches()
    with pytest.raises(pcd.PCDError) as err:
        pcd.batch_solve(ctx, bs, phis, _options(max_iterations=20000))
    # the start, three chunks of a pass and a refresh at most, the return of phi
    launches = L.pcd_kernel_launches() - before
    assert err.value.status == pcd._lib.PCD_TIMEOUT
    assert L.pcd_ctx_set_wait_limit(ctx.handle, 0, 0) == 0
    assert all(torch.equal(a, b) for a, b in zip(phis, starts))
    assert launches <= 8, launches
