"""The work that a user of this framework has it do, as cases that can be timed.

A caustic design spends its time in Poisson solves on grids of four times the
mesh's resolution, so most cases are solves: alone, on the device and through
the reference's host call, in FP64 and in mixed precision, with both stop
tests, from a zero guess, from the previous potential and from the network's
prediction; batched; and inside whole design steps.  The network's training
step is there too.  Sizes are those of the configurations in the tests and
the benchmark (grids of 64^2 to 4096^2, meshes of 128^2 and 1024^2, batches of
64 uneven grids, training batches of 32) and of meshes whose sides are no
power of two, whose grids are multiples of 4 but not of 8.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import poisson_caustic_design_gb300 as pcd
from poisson_caustic_design_gb300 import _lib, inputs, learned
from poisson_caustic_design_gb300.caustic_design import CausticDesign

_kept = {}


def _context():
    """One context and one network for the program, as the library asks for."""
    if "ctx" not in _kept:
        _kept["ctx"] = pcd.Context(0)
    return _kept["ctx"]


def _network():
    if "net" not in _kept:
        net = learned.UNet(_context(), resolution=64, max_batch=1)
        net.load(learned.default_weights_path(64))
        net.attach(_context())
        _kept["net"] = net
    return _kept["net"]


# ---- inputs ---------------------------------------------------------------

def _rhs(width, height, seed):
    """density - 1 with the mean removed: Gaussian mixtures and binary shapes
    (the two families of the benchmark) in turn, evaluated on the GPU."""
    rng = np.random.default_rng(seed)
    y = (torch.arange(height, device="cuda", dtype=torch.float64) + 0.5) / height
    x = (torch.arange(width, device="cuda", dtype=torch.float64) + 0.5) / width
    if seed % 2 == 0:
        rho = torch.full((height, width), 0.05, device="cuda", dtype=torch.float64)
        for _ in range(16):
            cx, cy = rng.uniform(0.1, 0.9, size=2)
            s, a = rng.uniform(0.03, 0.15), rng.uniform(0.2, 1.0)
            gy = a * torch.exp(-((y - cy) ** 2) / (2 * s * s))
            gx = torch.exp(-((x - cx) ** 2) / (2 * s * s))
            rho += gy[:, None] * gx[None, :]
    else:
        rho = torch.full((height, width), 0.02, device="cuda", dtype=torch.float64)
        for _ in range(20):
            cx, cy = rng.uniform(0.05, 0.95, size=2)
            if rng.uniform() < 0.5:
                r = rng.uniform(0.03, 0.15)
                rho[((y - cy) ** 2)[:, None] + ((x - cx) ** 2)[None, :] <= r * r] = 1.0
            else:
                hw, hh = rng.uniform(0.03, 0.15, size=2)
                rho[((y - cy).abs() <= hh)[:, None] & ((x - cx).abs() <= hw)[None, :]] = 1.0
    b = rho / rho.mean() - 1.0
    b = b - b.mean()
    return (b - b.mean()).contiguous()


def _exact_phi(b):
    """The mean-free solution of the Neumann problem, by the FFT of the even
    extension (whose periodic Laplacian is the Neumann one)."""
    h, w = b.shape
    t = torch.cat([b, b.flip(1)], 1)
    t = torch.cat([t, t.flip(0)], 0)
    f = torch.fft.rfft2(t)
    ky = torch.arange(2 * h, device=b.device, dtype=torch.float64)
    kx = torch.arange(f.shape[1], device=b.device, dtype=torch.float64)
    lam = (2 * torch.cos(math.pi * ky / h) - 2)[:, None] + (2 * torch.cos(math.pi * kx / w) - 2)[None, :]
    lam[0, 0] = 1.0
    f = f / lam
    f[0, 0] = 0.0
    phi = torch.fft.irfft2(f, s=t.shape)[:h, :w]
    return phi - phi.mean()


# ---- cases ----------------------------------------------------------------

def _solve(width, height, precision="mixed", stop="residual", start="zero", call="device", name=None):
    c = {"kind": "solve", "width": width, "height": height, "precision": precision, "stop": stop, "start": start,
         "call": call}
    return dict(c, name=name) if name else c


def _batch(count, largest, sizes_seed, name=None):
    c = {"kind": "batch", "count": count, "largest": largest, "sizes_seed": sizes_seed}
    return dict(c, name=name) if name else c


def _design(mesh_x, mesh_y, precision, heights, name=None):
    c = {"kind": "design", "mesh_x": mesh_x, "mesh_y": mesh_y, "precision": precision, "heights": heights}
    return dict(c, name=name) if name else c


def _train(batch, name=None):
    c = {"kind": "train", "batch": batch}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest solve of the tests and the benchmark's batch: a few hundred sweeps, latency
        _solve(64, 48, name="solve 64x48"),
        # the grid of a 63 x 47 mesh: a ragged width
        _solve(252, 188, name="solve 252x188"),
        # the benchmark's single solve, to relative residual 1e-6, in its three forms
        _solve(512, 512, name="solve 512"),
        _solve(512, 512, start="learned", name="solve 512 learned"),
        _solve(512, 512, precision="fp64", name="solve 512 fp64"),
        # the reference's call on host arrays with its own relaxation factor and stop
        _solve(256, 256, precision="fp64", stop="update", call="host", name="poisson_solver 256"),
        # a transport solve of a large design: the previous potential as the start, the reference's stop
        _solve(1024, 1024, stop="update", start="given", name="solve 1024 update"),
        # a single large grid, of a 512 x 375 mesh
        _solve(2048, 1500, name="solve 2048x1500"),
        # 64 uneven grids of 64^2 to 1024^2
        _batch(64, 1024, 17, name="batch 64"),
        # the full pipeline's steps at the 128^2 mesh with the reference's solves (FP64)
        _design(128, 128, "fp64", True, name="design 128"),
        # the largest configuration: 1024^2 mesh, 4096^2 grids, mixed precision
        _design(1024, 1024, "mixed", False, name="design 1024"),
        # a training step of the warm-start network at its documented batch
        _train(32, name="train 64x32"),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choices(["solve", "batch", "design", "train"], [8, 2, 2, 1])[0]
    if kind == "solve":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        top = 2048 if precision == "mixed" else 768
        # grids are four times a mesh; one in four is any size at all
        step = rng.choice([4, 4, 4, 1])
        width = int(_log_uniform(rng, 48, top)) // step * step
        height = min(top, max(48, int(width * rng.uniform(0.6, 1.6)))) // step * step
        call = "host" if precision == "fp64" and rng.random() < 0.4 else "device"
        start = rng.choice(["zero", "given", "learned"]) if precision == "mixed" else "zero"
        stop = "update" if call == "host" or start == "given" else rng.choice(["residual", "residual", "update"])
        return _solve(width, height, precision, stop, start, call)
    if kind == "batch":
        return _batch(rng.randint(4, 64), rng.choice([256, 512, 1024]), rng.randrange(1 << 20))
    if kind == "design":
        precision = rng.choice(["fp64", "mixed"])
        mesh = int(_log_uniform(rng, 32, 128 if precision == "fp64" else 512))
        return _design(mesh, max(24, int(mesh * rng.uniform(0.7, 1.0))), precision, rng.random() < 0.5)
    return _train(rng.randint(4, 48))


def _sides(case):
    rng = np.random.default_rng(case["sizes_seed"])
    sizes = [n for n in (64, 96, 128, 256, 512, 1024) if n <= case["largest"]]
    return [int(rng.choice(sizes)) for _ in range(case["count"])]


def _options(case):
    o = pcd.SolveOptions()
    if case["call"] == "host":
        return o
    o.omega = -1.0
    o.precision = pcd.PREC_MIXED if case["precision"] == "mixed" else pcd.PREC_FP64
    if case["stop"] == "residual":
        o.stop, o.tol = pcd.STOP_REL_RESIDUAL, 1e-6
    else:
        o.stop, o.tol = pcd.STOP_MAX_UPDATE, 1e-7
    o.warm_start = {"zero": 0, "given": 1, "learned": 2}[case["start"]]
    return o


def prepare(case, seed):
    ctx = _context()
    if case["kind"] == "solve":
        if case["start"] == "learned":
            _network()
        b = _rhs(case["width"], case["height"], seed)
        s = {"case": case, "opts": _options(case)}
        if case["call"] == "host":
            s["b"] = b.cpu().numpy()
            s["phi"] = np.zeros_like(s["b"])
            return s
        s["b"], s["phi"] = b, torch.zeros_like(b)
        if case["start"] == "given":
            # the potential of the step before: that of a nearby density
            s["guess"] = 0.9 * _exact_phi(b)
        return s
    if case["kind"] == "batch":
        bs = [_rhs(n, n, seed * 64 + i) for i, n in enumerate(_sides(case))]
        return {"case": case, "bs": bs, "phis": [torch.zeros_like(b) for b in bs]}
    if case["kind"] == "design":
        mx, my = case["mesh_x"], case["mesh_y"]
        mixed = case["precision"] == "mixed"
        opts = {}
        if mixed:
            opts = {"transport": pcd.SolveOptions(tol=1e-7, precision=pcd.PREC_MIXED, omega=-1.0),
                    "height_solve": pcd.SolveOptions(tol=1e-8, precision=pcd.PREC_MIXED, omega=-1.0)}
        d = CausticDesign(ctx, **opts)
        d.set_mesh_resolution(mx, my)
        d.set_domain_resolution(4 * mx, 4 * my)
        d.set_mesh_size(0.5, 0.5 * my / mx)
        d.set_lens_focal_length(1.5)
        d.set_lens_thickness(0.1)
        gray = inputs.gray_from_u8(inputs.gaussian_image(128, seed))
        return {"case": case, "design": d, "image": inputs.resize_nearest(gray, 4 * mx, 4 * my)}
    net = learned.UNet(ctx, resolution=64, max_batch=case["batch"], seed=7)
    x, t = [], []
    for i in range(case["batch"]):
        b = _rhs(64, 64, seed * 64 + i)
        sd = b.std()
        x.append((b / sd).float())
        t.append((_exact_phi(b) / (sd * 64 * 64)).float())
    return {"case": case, "net": net, "x": torch.stack(x), "t": torch.stack(t)}


def _remove_mean(phi):
    """A potential is defined up to a constant: programs that compare or train
    on potentials take its mean out."""
    stream = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.load().pcd_subtract_average_noalloc(phi.data_ptr(), phi.shape[1], phi.shape[0],
                                                        ctypes.c_void_p(stream)), "pcd_subtract_average_noalloc")


def run(state):
    case, ctx = state["case"], _context()
    if case["kind"] == "solve":
        b, phi = state["b"], state["phi"]
        if case["call"] == "host":
            phi.fill(0.0)
            pcd.poisson_solver(b, phi, case["width"], case["height"], 100000, 1e-7, 8)
            return phi - phi.mean()
        if case["start"] == "given":
            phi.copy_(state["guess"])
        ctx.solve_device(b, phi, state["opts"])
        _remove_mean(phi)
        return phi
    if case["kind"] == "batch":
        pcd.batch_solve(ctx, state["bs"], state["phis"], pcd.SolveOptions(stop=pcd.STOP_REL_RESIDUAL, tol=1e-6,
                                                                          omega=-1.0, warm_start=0))
        for p in state["phis"]:
            _remove_mean(p)
        return state["phis"]
    if case["kind"] == "design":
        d = state["design"]
        d.initialize_solvers(state["image"])
        out = {"step": d.perform_transport_iteration()}
        if case["heights"]:
            out["update"] = d.perform_height_map_iteration(0)
            out["source_points"] = d.source_points()
        out["target_points"] = d.target_points()
        return out
    net = state["net"]
    loss = net.train_step(state["x"], state["t"], 1e-3, 1e-5)
    return {"loss": loss, "gradients": net.grads()}


def exact(case, seed):
    """Potentials from the FFT; the pipeline's steps and the network's
    gradients (BF16 storage between its layers) have no such value."""
    if case["kind"] == "solve":
        phi = _exact_phi(_rhs(case["width"], case["height"], seed))
        return phi.cpu().numpy() if case["call"] == "host" else phi
    if case["kind"] == "batch":
        return [_exact_phi(_rhs(n, n, seed * 64 + i)) for i, n in enumerate(_sides(case))]
    return None


def _sweep_flops(cells, side, precision, stop):
    """Seven operations a cell and sweep; the sweeps of the relaxation at its
    optimal factor, in proportion to the longer side."""
    return 7.0 * cells * side * (5.0 if stop == "residual" else 5.5) * (2.0 if precision == "reference" else 1.0)


def work(case):
    if case["kind"] == "solve":
        cells = case["width"] * case["height"]
        side = max(case["width"], case["height"])
        return {"bytes": cells * (24 if case["start"] == "given" else 16),
                "flops": _sweep_flops(cells, side, "reference" if case["call"] == "host" else "", case["stop"])}
    if case["kind"] == "batch":
        sides = _sides(case)
        return {"bytes": sum(16 * n * n for n in sides),
                "flops": sum(_sweep_flops(n * n, n, "", "residual") for n in sides)}
    if case["kind"] == "design":
        n = case["mesh_x"] * case["mesh_y"]
        solves = 1.5 if case["heights"] else 1.0
        return {"bytes": 16 * n * 8 + n * 24 * (2 if case["heights"] else 1),
                "flops": solves * _sweep_flops(16 * n, 4 * max(case["mesh_x"], case["mesh_y"]),
                                               "reference" if case["precision"] == "fp64" else "", "update")}
    # every convolution forward, its data and its weight gradient, two operations a multiply-add
    flops = sum(3 * 2.0 * 9 * ci * co * (64 >> level) ** 2 for ci, co, level in learned.LAYERS) * case["batch"]
    n = learned.param_layout()[0][-1][1] + 1
    return {"bytes": case["batch"] * 2 * 64 * 64 * 4 + 5 * 4 * n, "flops": flops}
