"""Contexts of several host threads at once: the launches of one may not depend
on what another does between them."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,schedule,sizes,sweeps,solves", [
    (1, 0, (512, 256), 1600, 12),    # resident sweeps: a launch every 16 sweeps
    (0, 7, (512, 64), 8, 400),       # FP64 blocks: one launch a solve
    (0, 2, (256, 64), 8, 400),       # persistent bands
    (1, 3, (512, 384), 320, 40),     # one cluster
])
def test_threads_solve_grids_of_unlike_sizes(precision, schedule, sizes, sweeps, solves):
    """Two threads for each size, each with a context and a stream of its own: every
    solve does what it does alone, bit for bit."""
    import torch

    import poisson_caustic_design_gb300 as pcd

    o = pcd.SolveOptions(stop=pcd.STOP_REL_RESIDUAL, tol=0.0, max_iterations=sweeps, precision=precision,
                         omega=-1.0, warm_start=0, schedule=schedule, refine_every=16 if precision else 0)

    def solve(c, b, n):
        stream = torch.cuda.Stream()
        out = []
        with torch.cuda.stream(stream):
            phi = torch.zeros_like(b)
            for _ in range(n):
                st = c.solve_device(b, phi, o)
                assert st["sweeps"] == sweeps
                out.append(phi.clone())
        stream.synchronize()
        return out

    alone, bs, ctxs = [], [], []
    for n in sizes:
        b = torch.from_numpy(pcd.inputs.poisson_rhs(n, 3, "gaussian")).cuda()
        torch.cuda.synchronize()
        for _ in range(2):
            c = pcd.Context(0)
            ctxs.append(c)
            bs.append(b)
            alone.append(solve(c, b, 1)[0])
    failed = []

    def work(k):
        try:
            for phi in solve(ctxs[k], bs[k], solves):
                assert torch.equal(phi, alone[k])
        except Exception as e:  # handed on to the test's thread
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(ctxs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c in ctxs:
        c.close()
    assert not failed, failed
