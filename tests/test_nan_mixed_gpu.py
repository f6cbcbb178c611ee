"""NaN cells of b in mixed precision."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import poisson_caustic_design_gb300 as pcd

    c = pcd.Context(0)
    yield c
    c.close()


def test_batch_solved_at_the_start_with_a_nan_cell(ctx):
    """The norms of a batched solve run over the cells whose b is a number: a start that
    solves the grid ends it there, as it stands."""
    import torch

    import poisson_caustic_design_gb300 as pcd

    m, n = 96, 128
    y, x = torch.meshgrid(torch.arange(m, dtype=torch.float64), torch.arange(n, dtype=torch.float64), indexing="ij")
    phi = (torch.cos(y / 7.0) + torch.sin(x / 5.0)).cuda()
    pad = torch.nn.functional.pad(phi[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
    b = pad[:-2, 1:-1] + pad[2:, 1:-1] + pad[1:-1, :-2] + pad[1:-1, 2:] - 4.0 * phi
    b[40, 50] = float("nan")
    got = phi.clone()
    stats, _ = pcd.batch_solve(ctx, [b], [got], pcd.SolveOptions(stop=pcd.STOP_REL_RESIDUAL, tol=1e-6, omega=-1.0,
                                                                 max_iterations=500, precision=pcd.PREC_MIXED))
    assert stats[0]["converged"] and stats[0]["sweeps"] == 0 and stats[0]["rel_residual"] <= 1e-6
    assert torch.equal(got, phi)
