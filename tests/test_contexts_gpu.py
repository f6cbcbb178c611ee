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


@pytest.fixture
def stale_memory():
    """Small pieces of device memory that the next allocations get, not zero."""
    import ctypes

    import torch

    rt = ctypes.CDLL("libcudart.so." + torch.version.cuda.split(".")[0])
    ptrs = [ctypes.c_void_p() for _ in range(4096)]
    for p in ptrs:
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(512)) == 0
        assert rt.cudaMemset(p, 0x55, ctypes.c_size_t(512)) == 0
    torch.cuda.synchronize()
    for p in ptrs[::2]:
        assert rt.cudaFree(p) == 0
    yield
    torch.cuda.synchronize()
    for p in ptrs[1::2]:
        rt.cudaFree(p)


def _design(pcd, c):
    o = pcd.SolveOptions(tol=1e-7, precision=pcd.PREC_MIXED, omega=-1.0, max_iterations=20000)
    d = pcd.CausticDesign(c, transport=o, height_solve=o)
    d.set_mesh_resolution(32, 32)
    d.set_domain_resolution(128, 128)
    d.set_mesh_size(0.5, 0.5)
    d.set_lens_focal_length(1.5)
    d.set_lens_thickness(0.1)
    d.initialize_solvers(pcd.inputs.pipeline_image(32, 5))
    return d


def test_first_use_while_the_default_stream_is_busy(stale_memory):
    """A context's streams do not wait for the default stream, so its scratch has to be
    zero before they use it: the first mean removal, alone and in a design's step (whose
    solve has no solution otherwise and runs to its cap)."""
    import ctypes

    import torch

    import poisson_caustic_design_gb300 as pcd

    quiet, busy, designing = pcd.Context(0), pcd.Context(0), pcd.Context(0)
    expected = _design(pcd, quiet)
    step = expected.perform_transport_iteration()
    d = _design(pcd, designing)
    g = torch.rand(200, 300, dtype=torch.float64, device="cuda") + 1.0
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(1_000_000_000)  # half a second of the default stream
    st = pcd._lib.load().pcd_subtract_average_device(busy.handle, g.data_ptr(), 300, 200,
                                                     ctypes.c_void_p(stream.cuda_stream))
    assert st == 0
    stream.synchronize()
    mean = g.mean().item()
    torch.cuda._sleep(1_000_000_000)
    got = d.perform_transport_iteration()
    torch.cuda.synchronize()
    assert abs(mean) < 1e-12
    assert d.last_solve_stats["converged"]
    assert d.last_solve_stats["sweeps"] == expected.last_solve_stats["sweeps"] and got == step
    for x in (expected, d, quiet, busy, designing):
        x.close()
