"""Spacings far beyond the sweep cap ("never"): what the cap itself gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NEVER = 2**31 - 1


@pytest.fixture(scope="module")
def ctx():
    import poisson_caustic_design_gb300 as pcd

    c = pcd.Context(0)
    yield c
    c.close()


# estimate cycles on one tile and on many; persistent bands' chunks resident and
# on tile passes; tile passes
@pytest.mark.parametrize("n,m,schedule,stop,used,kw,cap", [
    (64, 48, 0, 1, 6, "check_every", 300), (256, 256, 0, 1, 6, "check_every", 300),
    (512, 300, 0, 1, 6, "refine_every", 300), (300, 260, 0, 0, 6, "check_every", 75),
    (1255, 1016, 0, 0, 2, "check_every", 75), (512, 512, 6, 0, 6, "refine_every", 75)])
def test_spacing_beyond_the_cap(ctx, n, m, schedule, stop, used, kw, cap):
    import poisson_caustic_design_gb300 as pcd

    b = pcd.inputs.poisson_rhs(n, 4, "gaussian", m=m)
    out = []
    for spacing in (cap, NEVER):
        phi = np.zeros_like(b)
        st = ctx.solve(b, phi, pcd.SolveOptions(stop=stop, tol=0.0, max_iterations=cap, omega=1.9, schedule=schedule,
                                                precision=pcd.PREC_MIXED, **{kw: spacing}))
        assert st["sweeps"] == cap and st["schedule_used"] == used
        out.append((phi, st["last_max_update"]))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


def test_batch_spacing_beyond_the_cap(ctx):
    import torch

    import poisson_caustic_design_gb300 as pcd

    bs = [torch.from_numpy(pcd.inputs.poisson_rhs(n, 4, "gaussian", m=m)).cuda() for m, n in [(161, 232), (96, 128)]]
    out = []
    for spacing in (43, NEVER):
        phis = [torch.zeros_like(b) for b in bs]
        stats, bst = pcd.batch_solve(ctx, bs, phis, pcd.SolveOptions(
            stop=pcd.STOP_REL_RESIDUAL, tol=1e-14, max_iterations=43, omega=1.9, refine_every=spacing,
            precision=pcd.PREC_MIXED))
        assert [s["sweeps"] for s in stats] == [43, 43] and bst["check_every"] == spacing
        out.append(phis)
    assert all(torch.equal(a, b) for a, b in zip(*out))
