"""NaN cells of b in mixed precision: AUTO finds them after it has started for a
grid without any, and goes on with the masked launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import poisson_caustic_design_gb300 as pcd

    c = pcd.Context(0)
    yield c
    c.close()


def _problem(n, m, ld):
    """b with a block of NaN cells, one at a corner and one on the last column, mean-free
    on the others, and a given start."""
    import torch

    import poisson_caustic_design_gb300 as pcd

    b = pcd.inputs.poisson_rhs(max(n, m), 9, "gaussian", m=max(n, m))[:m, :n].copy()
    b[m // 4:m // 4 + 5, n // 3:n // 3 + 7] = np.nan
    b[0, 0] = b[m // 2, n - 1] = np.nan
    b -= np.nanmean(b)
    start = 1e-2 * np.add.outer(np.cos(np.arange(m) / 7.0), np.sin(np.arange(n) / 5.0))
    out = []
    for a in (b, start):
        t = torch.zeros((m, ld), dtype=torch.float64, device="cuda")[:, :n]
        t.copy_(torch.from_numpy(a))
        out.append(t)
    return out


# resident (a whole and a partial lane column), below its sizes, tile passes, and
# a ragged width beyond the chip's registers
@pytest.mark.parametrize("n,m,ld", [(40, 30, 40), (41, 30, 44), (12, 30, 12), (1408, 1400, 1408), (1801, 1201, 1804)])
@pytest.mark.parametrize("stop", [0, 1])
@pytest.mark.parametrize("warm", [0, 1])
def test_auto_takes_the_masked_launches(ctx, n, m, ld, stop, warm):
    """The same bits as the masked launches asked for by name, and NaN where b is."""
    import torch

    import poisson_caustic_design_gb300 as pcd

    b, start = _problem(n, m, ld)
    out = []
    for sched in (1, 0):
        phi = torch.zeros((m, ld), dtype=torch.float64, device="cuda")[:, :n]
        phi.copy_(start)
        st = ctx.solve_device(b, phi, pcd.SolveOptions(stop=stop, tol=0.0, max_iterations=75, omega=1.8, warm_start=warm,
                                                       precision=pcd.PREC_MIXED, schedule=sched))
        assert st["sweeps"] == 75 and st["sweep_form"] == 0
        out.append((phi, st["rel_residual"], st["last_max_update"]))
    assert torch.equal(torch.isnan(out[1][0]), torch.isnan(b))
    assert torch.equal(torch.nan_to_num(out[0][0]), torch.nan_to_num(out[1][0]))
    assert out[0][1:] == out[1][1:]


@pytest.mark.parametrize("stop", [0, 1])
@pytest.mark.parametrize("warm", [0, 1])
def test_auto_with_nan_cells_reaches_the_fp64_solve(ctx, stop, warm):
    import torch

    import poisson_caustic_design_gb300 as pcd

    b, start = _problem(40, 30, 44)
    out = []
    for precision in (pcd.PREC_FP64, pcd.PREC_MIXED):
        phi = torch.zeros((30, 44), dtype=torch.float64, device="cuda")[:, :40]
        phi.copy_(start)
        st = ctx.solve_device(b, phi, pcd.SolveOptions(stop=stop, tol=1e-11, omega=-1.0, warm_start=warm,
                                                       precision=precision, max_iterations=20000))
        assert st["converged"]
        out.append(phi.cpu().numpy())
    m = ~np.isnan(out[0])
    a, c = (x[m] - x[m].mean() for x in out)
    assert np.abs(a - c).max() < 1e-7 * np.abs(a).max()


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
