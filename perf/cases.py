"""Workloads of the wave-propagation library and its learned corrector, as a
user's program runs them: one pass is one claw call over an output frame (from
the frame's start state, which the pass loads first), one inference pass of the
corrector or one of its training steps.

Inputs come from the seed alone.  Grids of a few thousand cells go in and out
as host arrays, as claw1ez / claw2ez hold them; larger ones are loaded and read
in place through the device view of q (``claw_q_device``), as the corrector's
own loops do, and a batch is loaded and read instance by instance from the
host.  ``exact`` restates each method in plain torch, in 64 bits.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from classic_b200 import problems
from classic_b200._lib import check
from classic_b200.corrector import LAYERS, ConvNet
from classic_b200.solver import BatchSolver, Solver

MINMOD, SUPERBEE, VANLEER, MC = "minmod", "superbee", "vanleer", "mc"
PULSE_BULK, PULSE_RHO = 4.0, 1.0  # the acoustics examples: c = 2, Z = 2
GAMMA = 1.4


def listed():
    return [
        # The 1D example at its configured size: one output frame of a small
        # grid (89 steps), host array in and out; latency per step counts.
        dict(name="line_800", kind="line", mx=800, limiter=MC, frame=0.1),
        # The annulus example at its test's size: a 2D grid far too small to
        # fill the GPU, with capacity, edge velocities and a periodic axis.
        dict(name="annulus_40x120", kind="annulus", mx=40, my=120, frame=0.25),
        # 2D radial acoustics at the configured 1024^2 in the default
        # arithmetic (the reference's order of operations).
        dict(name="radial_1024_fp64", kind="plane", mx=1024, my=1024, precision="fp64",
             limiter=MC, split="unsplit", bc="open", frame=0.03),
        # The headline: 4096^2, contracted FP64, one output frame (137 steps).
        dict(name="radial_4096_fma", kind="plane", mx=4096, my=4096, precision="fp64_fma",
             limiter=MC, split="unsplit", bc="open", frame=0.03),
        # An odd, oblong grid in FP32 with walls and another limiter.
        dict(name="radial_3001x1777_fp32", kind="plane", mx=3001, my=1777, precision="fp32",
             limiter=VANLEER, split="unsplit", bc="wall", frame=0.02),
        # Dimensional splitting in the default arithmetic, periodic in x.
        dict(name="strang_1501x1100_fp64", kind="plane", mx=1501, my=1100, precision="fp64",
             limiter=MC, split="strang", bc="periodic", frame=0.02),
        # The configured 3D run (256^3, two layers) in contracted FP64: the
        # most work of one call here.
        dict(name="layers_256_fma", kind="layers", mx=256, my=256, mz=256, precision="fp64_fma",
             limiter=MC, frame=0.1),
        # The same medium on a ragged box in FP32.
        dict(name="layers_161x130x147_fp32", kind="layers", mx=161, my=130, mz=147,
             precision="fp32", limiter=MC, frame=0.1),
        # ... and at 128^3 in the default arithmetic.
        dict(name="layers_128_fp64", kind="layers", mx=128, my=128, mz=128, precision="fp64",
             limiter=MC, frame=0.1),
        # A batched ensemble of uneven Euler grids, each with its own dt.
        dict(name="ensemble_16_fma", kind="ensemble", count=16, smallest=128, largest=384,
             sizes=7, precision="fp64_fma", limiter=MC, frame=0.06),
        # The corrector's inference on a batch of configured coarse grids.
        dict(name="corrector_8x256", kind="infer", images=8, h=256, w=256),
        # One training step of the corrector on a batch of crops.
        dict(name="train_16x64", kind="train", images=16, h=64, w=64),
    ]


def draw(rng):
    def span(lo, hi):  # log-uniform whole number
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["line", "annulus", "plane", "plane", "plane", "layers", "layers",
                       "ensemble", "infer", "train"])
    if kind == "line":
        return dict(kind=kind, mx=span(60, 1600), limiter=rng.choice([MINMOD, SUPERBEE, VANLEER, MC]),
                    frame=0.1)
    if kind == "annulus":
        return dict(kind=kind, mx=span(20, 300), my=span(60, 900), frame=0.1)
    if kind == "plane":
        return dict(kind=kind, mx=span(100, 3200), my=span(100, 3200),
                    precision=rng.choice(["fp64", "fp64_fma", "fp32"]),
                    limiter=rng.choice([MINMOD, SUPERBEE, VANLEER, MC]),
                    split=rng.choice(["unsplit", "unsplit", "godunov", "strang"]),
                    bc=rng.choice(["open", "wall", "periodic"]), frame=0.02)
    if kind == "layers":
        return dict(kind=kind, mx=span(24, 200), my=span(24, 200), mz=span(24, 200),
                    precision=rng.choice(["fp64", "fp64_fma", "fp32"]),
                    limiter=rng.choice([VANLEER, MC]), frame=0.05)
    if kind == "ensemble":
        lo = span(48, 160)
        return dict(kind=kind, count=span(2, 24), smallest=lo, largest=span(lo, 384),
                    sizes=rng.randrange(1000), precision=rng.choice(["fp64", "fp64_fma"]),
                    limiter=MC, frame=0.04)
    if kind == "infer":
        return dict(kind=kind, images=span(1, 12), h=16 * rng.randint(2, 16), w=16 * rng.randint(2, 16))
    return dict(kind=kind, images=span(2, 24), h=16 * rng.randint(2, 6), w=16 * rng.randint(2, 6))


# ------------------------------------------------------------------ inputs ---
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _centres(lo, hi, n):
    return lo + (torch.arange(1, n + 1, dtype=torch.float64, device=_device()) - 0.5) * ((hi - lo) / n)


def _line_q0(case, seed):
    r = np.random.default_rng(seed)
    x = -1.0 + (np.arange(case["mx"]) + 0.5) * (2.0 / case["mx"])
    q = np.zeros((2, case["mx"]))
    q[0] = r.uniform(0.5, 1.5) * np.exp(-100.0 * (x - r.uniform(0.1, 0.4)) ** 2)
    return q


def _annulus(case, seed):
    """(rundata, params, q0, aux): the example's mapping and edge velocities,
    two Gaussians of seeded strength and place."""
    rd, _, params, _, aux = problems.advection_2d_annulus(mx=case["mx"], my=case["my"])
    g = np.random.default_rng(seed)
    r = 0.2 + (np.arange(case["mx"]) + 0.5) * (0.8 / case["mx"])
    th = (np.arange(case["my"]) + 0.5) * (2.0 * np.pi / case["my"])
    x, y = r[None, :] * np.cos(th)[:, None], r[None, :] * np.sin(th)[:, None]
    q = np.zeros((1,) + x.shape)
    for sign in (1.0, -1.0):
        a, x0, y0 = sign * g.uniform(0.7, 1.3), -0.5 * sign + g.uniform(-0.1, 0.1), g.uniform(-0.1, 0.1)
        q[0] += a * np.exp(-40.0 * ((x - x0) ** 2 + (y - y0) ** 2))
    return rd, params, q, aux


BCS = {"open": (["extrap", "extrap"], ["extrap", "extrap"]),
       "wall": (["wall", "extrap"], ["extrap", "wall"]),
       "periodic": (["periodic", "extrap"], ["periodic", "extrap"])}


def _plane_q0(case, seed):
    """The radial ring of the configured run, with a seeded centre, radius and
    strength, in the storage type of the run."""
    g = np.random.default_rng(seed)
    x, y = _centres(-1.0, 1.0, case["mx"]), _centres(-1.0, 1.0, case["my"])
    r = torch.hypot(x[None, :] - g.uniform(-0.2, 0.2), y[:, None] - g.uniform(-0.2, 0.2))
    r0, a = g.uniform(0.3, 0.6), g.uniform(0.7, 1.3)
    q = torch.zeros((3, case["my"], case["mx"]), dtype=torch.float64, device=_device())
    q[0] = 1.0 + a * torch.where((r - r0).abs() < 0.1, torch.cos(math.pi * (r - r0) / 0.1), 0.0)
    return q.float() if case["precision"] == "fp32" else q


def _layers_q0(case, seed):
    g = np.random.default_rng(seed)
    x, y, z = (_centres(-1.0, 1.0, case[k]) for k in ("mx", "my", "mz"))
    c = g.uniform([-0.3, -0.3, -0.5], [0.3, 0.3, -0.2])
    r2 = ((x - c[0]) ** 2)[None, None, :] + ((y - c[1]) ** 2)[None, :, None] + ((z - c[2]) ** 2)[:, None, None]
    q = torch.zeros((4, case["mz"], case["my"], case["mx"]), dtype=torch.float64, device=_device())
    q[0] = g.uniform(0.7, 1.3) * torch.exp(-80.0 * r2)
    return q.float() if case["precision"] == "fp32" else q


def _layers_aux(case):
    """(Z, c) per cell with two ghost layers: rho, K = 1, 1 below z = 0 and 4, 2 above."""
    z = -1.0 + (np.arange(-1, case["mz"] + 3) - 0.5) * (2.0 / case["mz"])
    aux = np.empty((2, case["mz"] + 4, case["my"] + 4, case["mx"] + 4))
    aux[0] = np.where(z < 0.0, 1.0, math.sqrt(8.0))[:, None, None]
    aux[1] = np.where(z < 0.0, 1.0, math.sqrt(0.5))[:, None, None]
    return aux


def _sizes(case):
    g = np.random.default_rng(case["sizes"])
    lo, hi = math.log(case["smallest"]), math.log(case["largest"])
    return [(int(round(math.exp(g.uniform(lo, hi)))),) * 2 for _ in range(case["count"])]


def _quadrants(seed, k, mx, my):
    """Four-quadrant Riemann data of one instance, the configured family within
    the ranges that stay physical in every instance (p from 0.4, |u|, |v| to 0.5)."""
    g = np.random.default_rng([seed, k])
    rho, p = g.uniform(0.5, 2.0, 4), g.uniform(0.4, 1.5, 4)
    u, v = g.uniform(-0.5, 0.5, 4), g.uniform(-0.5, 0.5, 4)
    xs, ys = g.uniform(0.3, 0.7, 2)
    x, y = (np.arange(mx) + 0.5) / mx, (np.arange(my) + 0.5) / my
    quad = (x >= xs).astype(int)[None, :] + 2 * (y >= ys).astype(int)[:, None]
    prim = np.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)])
    return np.ascontiguousarray(prim[:, quad])


def _weights(seed):
    g = np.random.default_rng(seed)
    w, b = [], []
    for k, (cin, cout, act) in enumerate(LAYERS):
        a = g.standard_normal((cout, 9, cin)) * math.sqrt((2.0 if act else 0.5) / (9 * cin))
        if k == 0:
            a[:, :, 8:] = 0.0  # 8 of the 16 input channels are used
        if k == len(LAYERS) - 1:
            a[4:] = 0.0        # and 4 of the 16 outputs
        w.append(a.astype(np.float32))
        b.append((0.05 * g.standard_normal(cout) * (np.arange(cout) < (4 if not act else cout))).astype(np.float32))
    return {"w": w, "b": b}


def _images(case, seed):
    """Normalised features (8 of 16 channels) and, for training, targets whose
    crop margin is masked out with NaN, as the training loop masks it."""
    g = torch.Generator(device=_device()).manual_seed(seed)
    n, h, w = case["images"], case["h"], case["w"]
    x = torch.zeros((n, h, w, 16), dtype=torch.bfloat16, device=_device())
    x[..., :8] = torch.randn((n, h, w, 8), generator=g, device=_device()).to(torch.bfloat16)
    t = torch.randn((n, h, w, 4), generator=g, device=_device())
    t[:, :5] = float("nan")
    t[:, :, -5:] = float("nan")
    return x, t


def _spacing(case):
    return [2.0 / case[k] for k in ("mx", "my", "mz") if k in case]


def _dt0(case):
    """The time step a run in progress hands to its next frame."""
    if case["kind"] == "annulus":
        return 0.9 / (2.0 * math.pi * case["my"] / (2.0 * math.pi))
    c = 1.0 if case["kind"] == "layers" else math.sqrt(PULSE_BULK / PULSE_RHO)
    return 0.9 * min(_spacing(case)) / c


# ----------------------------------------------------------------- prepare ---
def _config(case):
    kind = case["kind"]
    if kind == "line":
        rd, solver, params, _, _ = problems.acoustics_1d_config(mx=case["mx"])
        rd.clawdata.limiter = [case["limiter"]] * 2
    elif kind == "plane":
        rd, solver, params, _, _ = problems.radial_acoustics_2d(n=8, limiter=case["limiter"])
        cd = rd.clawdata
        cd.num_cells, cd.dimensional_split = [case["mx"], case["my"]], case["split"]
        cd.bc_lower, cd.bc_upper = (list(b) for b in BCS[case["bc"]])
    else:
        rd, solver, params, _, _ = problems.heterogeneous_acoustics_3d(n=4, limiter=case["limiter"])
        rd.clawdata.num_cells = [case["mx"], case["my"], case["mz"]]
    return rd, solver, params


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, dt=_dt0(case) if kind in ("line", "annulus", "plane", "layers") else None)
    if kind == "line":
        rd, solver, params = _config(case)
        st.update(solver=Solver(rd, solver, params), q0=_line_q0(case, seed))
    elif kind == "annulus":
        rd, params, q0, aux = _annulus(case, seed)
        st.update(solver=Solver(rd, "vc_advection_2d", params), q0=q0)
        st["solver"].set_aux(aux)
    elif kind in ("plane", "layers"):
        rd, solver, params = _config(case)
        st["solver"] = Solver(rd, solver, params, precision=case["precision"])
        if kind == "layers":
            st["solver"].set_aux(_layers_aux(case))
        st["q0"] = (_plane_q0 if kind == "plane" else _layers_q0)(case, seed)
    elif kind == "ensemble":
        rds = []
        for mx, my in _sizes(case):
            rds.append(problems.euler_quadrants(shape=(4, 4), limiter=case["limiter"])[0])
            rds[-1].clawdata.num_cells = [mx, my]
        st["batch"] = BatchSolver(rds, "euler_roe_2d", {"gamma": GAMMA}, precision=case["precision"])
        st["q0"] = [_quadrants(seed, k, mx, my) for k, (mx, my) in enumerate(_sizes(case))]
        st["dt"] = [0.2 / max(s) for s in _sizes(case)]
    else:
        st["net"] = ConvNet(seed=0)
        st["net"].load(_weights(seed))
        st["x"], st["target"] = _images(case, seed)
    return st


# --------------------------------------------------------------------- run ---
class _View:
    """A device array that the library owns, for torch.as_tensor; the tensor
    keeps this object, and with it the owner of the memory, alive."""

    def __init__(self, owner, ptr, shape, strides, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "strides": strides, "typestr": typestr,
                                         "data": (ptr, False), "version": 3}


def _q_device(solver):
    """The solver's current q on the device, as a tensor of the grid's shape."""
    ptr, es = ctypes.c_void_p(), ctypes.c_int()
    ld, fp = ctypes.c_longlong(), ctypes.c_longlong()
    check(solver.lib.claw_q_device(solver._h, ctypes.byref(ptr), ctypes.byref(es), ctypes.byref(ld),
                                   ctypes.byref(fp)), "claw_q_device")
    shape = solver.q_shape
    rows = [ld.value] if len(shape) == 3 else [ld.value * shape[2], ld.value]
    strides = tuple(es.value * s for s in [fp.value] + rows + [1])
    return torch.as_tensor(_View(solver, ptr.value, shape, strides, "<f%d" % es.value), device="cuda")


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("line", "annulus"):
        s = state["solver"]
        s.set_q(state["q0"])
        info, st = s.advance(0.0, case["frame"], state["dt"])
        return {"q": s.get_q(), "dt": st["dt_next"], "steps": st["steps_taken"]}
    if kind in ("plane", "layers"):
        s = state["solver"]
        _q_device(s).copy_(state["q0"])
        torch.cuda.current_stream().synchronize()  # the solver's stream does not wait for torch's
        info, st = s.advance(0.0, case["frame"], state["dt"])
        return {"q": _q_device(s), "dt": st["dt_next"], "steps": st["steps_taken"]}
    if kind == "ensemble":
        b = state["batch"]
        for k, q in enumerate(state["q0"]):
            b.set_q(k, q)
        info, sts = b.advance(0.0, case["frame"], state["dt"])
        return {"q": [b.get_q(k) for k in range(b.count)], "dt": np.array([s["dt_next"] for s in sts]),
                "steps": np.array([s["steps_taken"] for s in sts])}
    net = state["net"]
    if kind == "infer":
        return net.forward(state["x"])[..., :4]
    pred = net.forward(state["x"], train=True)
    dy, loss = net.loss_grad(pred, state["target"])
    net.backward(dy)
    net.adam(lr=1e-3)
    return {"loss": loss, "gw": list(net.gw), "gb": list(net.gb), "w": list(net.w32)}


# -------------------------------------------------------------------- work ---
def _steps(case):
    return max(1, math.ceil(case["frame"] / _dt0(case)))


def work(case):
    """Per step each field read and written once and the coefficients read once
    (q is the state a step cannot avoid touching); the floating-point work is
    that of the method in its shortest form, per cell and step."""
    kind = case["kind"]
    if kind in ("line", "annulus", "plane", "layers"):
        cells = math.prod(_cells(case))
        size = 4 if case.get("precision") == "fp32" else 8
        fields, coeffs, flops = {"line": (2, 0, 40), "annulus": (1, 3, 60), "plane": (3, 0, 110),
                                 "layers": (4, 2, 700)}[kind]
        n = cells * _steps(case)
        return {"bytes": float(n * size * (2 * fields + coeffs)), "flops": float(n * flops)}
    if kind == "ensemble":
        n = sum(mx * my * max(1, math.ceil(case["frame"] * max(mx, my) / 0.3)) for mx, my in _sizes(case))
        return {"bytes": float(n * 64), "flops": float(n * 1500)}
    pixels = case["images"] * case["h"] * case["w"]
    macs = sum(9 * cin * cout for cin, cout, _ in LAYERS)
    if kind == "infer":
        return {"bytes": float(pixels * (16 * 2 + 4 * 4)), "flops": float(2 * macs * pixels)}
    data_grad = sum(9 * cin * cout for cin, cout, _ in LAYERS[1:])
    # forward, weight and data gradients; every activation written and read once
    return {"bytes": float(pixels * (16 * 2 + 4 * 4 + 2 * 4 * 32 * 2)), "flops": float(2 * (2 * macs + data_grad) * pixels)}


def _cells(case):
    return [case[k] for k in ("mz", "my", "mx") if k in case]


# ------------------------------------------------------------------- exact ---
def exact(case, seed):
    kind = case["kind"]
    if kind == "line":
        q, dt = _claw(case, lambda q, dt: _line_step(q, dt, 2.0 / case["mx"], case["limiter"]),
                      torch.from_numpy(_line_q0(case, seed)).to(_device()))
    elif kind == "annulus":
        _, _, q0, aux = _annulus(case, seed)
        aux = torch.from_numpy(aux).to(_device())
        d = (0.8 / case["mx"], 2.0 * math.pi / case["my"])
        bc = ((1, 1), (2, 2))
        q, dt = _claw(case, lambda q, dt: _step2(_Edges(), q, aux, 3, dt, d, [VANLEER], bc, "unsplit"),
                      torch.from_numpy(q0).to(_device()))
    elif kind == "plane":
        codes = {"extrap": 1, "periodic": 2, "wall": 3}
        lo, hi = BCS[case["bc"]]
        bc = tuple((codes[lo[k]], codes[hi[k]]) for k in range(2))
        q, dt = _claw(case, lambda q, dt: _step2(_Sound(), q, None, 0, dt, _spacing(case),
                                                 [case["limiter"]] * 2, bc, case["split"]),
                      _plane_q0(case, seed).double())
    elif kind == "layers":
        aux = torch.from_numpy(_layers_aux(case)).to(_device())
        q, dt = _claw(case, lambda q, dt: _step3(q, aux, dt, _spacing(case), case["limiter"]),
                      _layers_q0(case, seed).double())
    elif kind == "ensemble":
        if sum(work(case).values()) > 3e12:
            return None
        qs, dts = [], []
        for k, (mx, my) in enumerate(_sizes(case)):
            step = lambda q, dt: _step2(_Gas(), q, None, 0, dt, (1.0 / mx, 1.0 / my),  # noqa: E731
                                        [case["limiter"]] * 3, ((1, 1), (1, 1)), "unsplit")
            q, dt = _claw(case, step, torch.from_numpy(_quadrants(seed, k, mx, my)).to(_device()),
                          0.2 / max(mx, my))
            qs.append(q.cpu().numpy())
            dts.append(dt)
        return {"q": qs, "dt": np.array(dts), "steps": None}
    else:
        return _net_exact(case, seed)
    return {"q": q.cpu().numpy() if kind in ("line", "annulus") else q, "dt": dt, "steps": None}


def _claw(case, step, q, dt=None):
    """claw2's loop over one frame: accept up to Courant number 1, aim at 0.9."""
    t, tend = 0.0, case["frame"]
    dt = min(_dt0(case) if dt is None else dt, tend)
    while t < tend:
        qn, cfl = step(q, dt)
        if cfl <= 1.0:
            q, t = qn, t + dt
        dt = dt * 0.9 / cfl
        if t < tend and t + dt > tend:
            dt = tend - t
    return q, dt


def _phi(name, r):
    if name == MINMOD:
        return torch.clamp(r, 0.0, 1.0)
    if name == SUPERBEE:
        return torch.maximum(torch.clamp(2.0 * r, 0.0, 1.0), torch.clamp(r, 0.0, 2.0))
    if name == VANLEER:
        return (r + r.abs()) / (1.0 + r.abs())
    return torch.clamp(torch.minimum(torch.minimum(0.5 * (1.0 + r), 2.0 * r), torch.full_like(r, 2.0)), min=0.0)


def _limited(w, s, name):
    """Wave w[m, ..., interfaces] limited against its upwind neighbour, on the
    interfaces that have both."""
    own = w[..., 1:-1]
    norm = (own * own).sum(0)
    up = torch.where(s[..., 1:-1] > 0.0, (own * w[..., :-2]).sum(0), (own * w[..., 2:]).sum(0))
    phi = _phi(name, up / torch.where(norm == 0.0, torch.ones_like(norm), norm))
    return torch.where(norm == 0.0, torch.ones_like(phi), phi) * own


def _pad(q, bc):
    """Two ghost cells per side, axis by axis from x: 1 extrapolation, 2
    periodic, 3 wall (the axis' velocity changes sign)."""
    for axis, sides in enumerate(bc):
        dim, n = q.dim() - 1 - axis, q.shape[q.dim() - 1 - axis]
        parts = []
        for side, code in enumerate(sides):
            at = {1: [0, 0] if side == 0 else [n - 1, n - 1], 2: [n - 2, n - 1] if side == 0 else [0, 1],
                  3: [1, 0] if side == 0 else [n - 1, n - 2]}[code]
            g = q.index_select(dim, torch.tensor(at, device=q.device))
            if code == 3:
                g[1 + axis] = -g[1 + axis]
            parts.append(g)
        q = torch.cat([parts[0], q, parts[1]], dim)
    return q


def _line_step(q, dt, dx, limiter):
    z = c = 2.0
    p = torch.cat([q.flip(1)[:, -2:] * torch.tensor([[1.0], [-1.0]], device=q.device), q, q[:, -1:], q[:, -1:]], 1)
    d = p[:, 1:] - p[:, :-1]
    a1, a2 = (z * d[1] - d[0]) / (2.0 * z), (z * d[1] + d[0]) / (2.0 * z)
    w1, w2 = torch.stack([-z * a1, a1]), torch.stack([z * a2, a2])
    f = sum(0.5 * c * (1.0 - c * dt / dx) * _limited(w, s * torch.ones_like(a1), limiter)
            for w, s in ((w1, -c), (w2, c)))
    qn = q - dt / dx * (c * w2[:, 1:-2] - c * w1[:, 2:-1]) - dt / dx * (f[:, 1:] - f[:, :-1])
    return qn, c * dt / dx


class _Sound:
    """Constant-coefficient acoustics, q = (p, u, v)."""
    z = c = 2.0

    def normal(self, ixy, ql, qr, aux):
        dp, du = qr[0] - ql[0], qr[ixy] - ql[ixy]
        zero = torch.zeros_like(dp)
        out = []
        for a, s in (((self.z * du - dp) / (2.0 * self.z), -self.c), ((self.z * du + dp) / (2.0 * self.z), self.c)):
            w = [math.copysign(self.z, s) * a, zero, zero]
            w[ixy] = a
            out.append((torch.stack(w), s * torch.ones_like(dp)))
        return [o[0] for o in out], [o[1] for o in out], -self.c * out[0][0], self.c * out[1][0]

    def across(self, ixy, imp, ql, qr, aux, f):
        iv = 3 - ixy
        zero = torch.zeros_like(f[0])
        out = []
        for a, s in (((self.z * f[iv] - f[0]) / (2.0 * self.z), -1.0), ((self.z * f[iv] + f[0]) / (2.0 * self.z), 1.0)):
            w = [self.c * self.z * a, zero, zero]
            w[iv] = s * self.c * a
            out.append(torch.stack(w))
        return out


class _Edges:
    """Advection with edge velocities, aux = (u at the left, v at the bottom, capacity)."""

    def normal(self, ixy, ql, qr, aux):
        s = aux[ixy - 1, 1:-1, 1:]
        w = qr - ql
        return [w], [s], torch.clamp(s, max=0.0) * w, torch.clamp(s, min=0.0) * w

    def across(self, ixy, imp, ql, qr, aux, f):
        v = aux[2 - ixy, :, 1:-2] if imp == 1 else aux[2 - ixy, :, 2:-1]
        return [torch.clamp(v[1:-1], max=0.0) * f, torch.clamp(v[2:], min=0.0) * f]


class _Gas:
    """Euler, Roe's solver with Harten and Hyman's entropy fix."""

    def _roe(self, ixy, ql, qr):
        g1, (mu, mv) = GAMMA - 1.0, (ixy, 3 - ixy)
        sl, sr = torch.sqrt(ql[0]), torch.sqrt(qr[0])
        pl = g1 * (ql[3] - 0.5 * (ql[1] ** 2 + ql[2] ** 2) / ql[0])
        pr = g1 * (qr[3] - 0.5 * (qr[1] ** 2 + qr[2] ** 2) / qr[0])
        mean = lambda a, b: (a / sl + b / sr) / (sl + sr)  # noqa: E731
        u, v, h = mean(ql[mu], qr[mu]), mean(ql[mv], qr[mv]), mean(ql[3] + pl, qr[3] + pr)
        a2 = g1 * (h - 0.5 * (u * u + v * v))
        return u, v, h, torch.sqrt(a2), g1 / a2

    def _waves(self, mu, mv, d, u, v, h, a, g1a2):
        """Eigenvectors along the axis of mu, where u is the Roe velocity."""
        a3 = g1a2 * ((h - u * u - v * v) * d[0] + u * d[mu] + v * d[mv] - d[3])
        a2 = d[mv] - v * d[0]
        a4 = (d[mu] + (a - u) * d[0] - a * a3) / (2.0 * a)
        a1 = d[0] - a3 - a4
        ws = []
        for rho, mom, tan, en in ((a1, a1 * (u - a), a1 * v, a1 * (h - u * a)),
                                  (a3, a3 * u, a3 * v + a2, a3 * 0.5 * (u * u + v * v) + a2 * v),
                                  (a4, a4 * (u + a), a4 * v, a4 * (h + u * a))):
            w = [rho, None, None, en]
            w[mu], w[mv] = mom, tan
            ws.append(torch.stack(w))
        return ws, [u - a, u, u + a]

    @staticmethod
    def _state(q, mu):
        p = (GAMMA - 1.0) * (q[3] - 0.5 * (q[1] ** 2 + q[2] ** 2) / q[0])
        return q[mu] / q[0], torch.sqrt(GAMMA * p / q[0])

    def normal(self, ixy, ql, qr, aux):
        mu, mv = ixy, 3 - ixy
        w, s = self._waves(mu, mv, qr - ql, *self._roe(ixy, ql, qr))
        zero = torch.zeros_like(s[0])

        def share(sa, sb, speed):  # of a wave between the speeds sa and sb of its two sides
            mix = sa * (sb - speed) / (sb - sa)
            return torch.where((sa < 0.0) & (sb > 0.0), mix, torch.clamp(speed, max=0.0)), mix

        u, c = self._state(ql, mu)
        s0 = u - c
        u, c = self._state(ql + w[0], mu)
        f1, _ = share(s0, u - c, s[0])
        u, c = self._state(qr, mu)
        s3 = u + c
        u, c = self._state(qr - w[2], mu)
        s2 = u + c
        f3 = torch.where((s2 < 0.0) & (s3 > 0.0), s2 * (s3 - s[2]) / (s3 - s2), torch.clamp(s[2], max=0.0))
        am = f1 * w[0] + torch.where(s[1] < 0.0, s[1] * w[1] + f3 * w[2], zero)
        am = torch.where((s0 >= 0.0) & (s[0] > 0.0), zero, am)
        return w, s, am, s[0] * w[0] + s[1] * w[1] + s[2] * w[2] - am

    def across(self, ixy, imp, ql, qr, aux, f):
        u, v, h, a, g1a2 = self._roe(ixy, ql, qr)
        w, s = self._waves(3 - ixy, ixy, f, v, u, h, a, g1a2)
        return [sum(torch.clamp(x, max=0.0) * y for x, y in zip(s, w)),
                sum(torch.clamp(x, min=0.0) * y for x, y in zip(s, w))]


def _flux2(system, ixy, q, aux, capa, dtd, limiters, transverse):
    """flux2 over every slice along the last axis of q[m, across, along], ghost
    cells included, on the slices 1..-1: the increments (own, flux at the
    cell's lower and upper interface, transverse fluxes down and up) of the
    interior cells of each slice, and the Courant number."""
    mid = q[:, 1:-1]
    ql, qr = mid[..., :-1], mid[..., 1:]
    w, s, am, ap = system.normal(ixy, ql, qr, aux)
    d = dtd / aux[capa - 1, 1:-1] if capa else torch.full_like(mid[0], dtd)
    inner = slice(1, -1)
    cfl = max(float(torch.maximum(d[..., 2:-1] * x[..., inner], -d[..., 1:-2] * x[..., inner]).max()) for x in s)
    ave = 0.5 * (d[..., 1:-2] + d[..., 2:-1])
    cq = 0.0
    for x, y, name in zip(w, s, limiters):
        sp = y[..., inner].abs()
        cq = cq + sp * (1.0 - sp * ave) * _limited(x, y, name)
    am, ap = am[..., inner], ap[..., inner]
    dc = d[..., 2:-2]
    own = -dc * (ap[..., :-1] + am[..., 1:])
    if not transverse:
        return own, 0.5 * cq, None, None, cfl
    ql, qr = ql[..., inner], qr[..., inner]
    left = system.across(ixy, 1, ql, qr, aux, am + cq)
    right = system.across(ixy, 2, ql, qr, aux, ap - cq)
    down, up = (-0.5 * dc * (a[..., 1:] + b[..., :-1]) for a, b in zip(left, right))
    return own, 0.5 * cq, down, up, cfl


def _step2(system, q, aux, capa, dt, d, limiters, bc, split):
    turn = lambda a: a.transpose(-1, -2).contiguous()  # noqa: E731
    p = _pad(q, bc)
    if split == "unsplit":
        out, cfls = q.clone(), []
        for ixy in (1, 2):
            side = p if ixy == 1 else turn(p)
            a = aux if ixy == 1 or aux is None else turn(aux)
            k = a[capa - 1, 2:-2, 2:-2] if capa else 1.0
            tn, tt = (dt / d[0], dt / d[1]) if ixy == 1 else (dt / d[1], dt / d[0])
            own, f, down, up, cfl = _flux2(system, ixy, side, a, capa, tn, limiters, True)
            inc = own[:, 1:-1] - tn * (f[:, 1:-1, 1:] - f[:, 1:-1, :-1]) / k \
                - tt * (up[:, 1:-1] - down[:, 1:-1] + down[:, 2:] - up[:, :-2]) / k
            out = out + (inc if ixy == 1 else inc.transpose(-1, -2))
            cfls.append(cfl)
        return out, max(cfls)
    # dimsp2: sweeps over the ghost slices too; ghost cells keep bc2's values
    # along their own sweep
    sweeps = [(1, dt), (2, dt)] if split == "godunov" else [(1, 0.5 * dt), (2, dt), (1, 0.5 * dt)]
    cfls = []
    for ixy, h in sweeps:
        side = p if ixy == 1 else turn(p)
        wide = torch.cat([side[:, :1], side, side[:, -1:]], 1)  # _flux2 drops a slice each side
        tn = h / d[ixy - 1]
        own, f, _, _, cfl = _flux2(system, ixy, wide, None, 0, tn, limiters, False)
        side = side.clone()
        side[..., 2:-2] += own - tn * (f[..., 1:] - f[..., :-1])
        p = side if ixy == 1 else turn(side)
        cfls.append(cfl)
    return p[:, 2:-2, 2:-2].contiguous(), max(cfls)


def _step3(q, aux, dt, d, limiter):
    """step3 with transverse code 22 for variable-coefficient acoustics.  Every
    transverse term is linear in two numbers per cell and sweep: x (the first
    splits) and y (what is split twice), so the corrections are face fluxes of
    x and mixed differences of edge fluxes of y."""
    p = _pad(q, ((1, 1), (1, 1), (3, 1)))
    out, cfls = q.clone(), []
    for n in range(3):
        e1, e2 = ((1, 2), (0, 2), (0, 1))[n]
        lay = lambda a: a.permute(*[2 - k for k in (e2, e1, n)])  # noqa: E731  [e2, e1, n]
        tn, t1, t2 = dt / d[n], dt / d[e1], dt / d[e2]
        pr, un = lay(p[0])[1:-1, 1:-1], lay(p[1 + n])[1:-1, 1:-1]
        z, c = lay(aux[0])[1:-1, 1:-1], lay(aux[1])[1:-1, 1:-1]
        zl, zr, cl, cr = z[..., :-1], z[..., 1:], c[..., :-1], c[..., 1:]
        dp, du = pr[..., 1:] - pr[..., :-1], un[..., 1:] - un[..., :-1]
        a1, a2 = (zr * du - dp) / (zl + zr), (zl * du + dp) / (zl + zr)
        w1, w2 = torch.stack([-zl * a1, a1]), torch.stack([zr * a2, a2])
        cfls.append(tn * float(c.max()))
        cq = 0.0
        for w, s in ((w1, -cl), (w2, cr)):
            sp = s[..., 1:-1].abs()
            cq = cq + 0.5 * sp * (1.0 - sp * tn) * _limited(w, s, limiter)
        am, ap = (-cl * w1)[..., 1:-1], (cr * w2)[..., 1:-1]
        total, diff = am[..., 1:] + ap[..., :-1], cq[..., 1:] - cq[..., :-1]
        inner = (slice(1, -1), slice(1, -1))
        inc = [torch.zeros_like(diff[0][inner]) for _ in range(4)]
        inc[0] = inc[0] - tn * (total[0] + diff[0])[inner]
        inc[1 + n] = inc[1 + n] - tn * (total[1] + diff[1])[inner]
        x = -0.5 * tn * total[0] - tn * diff[0]
        y = total[0] + 3.0 * diff[0]
        z, c = z[..., 2:-2], c[..., 2:-2]
        for ax, te, tw, comp in ((1, t1, t2, 1 + e1), (0, t2, t1, 1 + e2)):
            # turned so that the split axis is the second one
            f = (lambda a: a) if ax == 1 else (lambda a: a.transpose(0, 1))
            fx, fy, fz, fc = f(x), f(y), f(z), f(c)

            def faces(v, k):  # (pressure, velocity) of v split at the faces along axis 1 of layer(s) k
                zz, cc = fz[k], fc[k]
                r = 1.0 / (zz[:, 1:] + zz[:, :-1])
                hi, lo = cc[:, 1:] * r * v[:, :-1], cc[:, :-1] * r * v[:, 1:]
                return zz[:, 1:] * hi - zz[:, :-1] * lo, hi + lo

            flux = [a[1:-1] for a in faces(fx, slice(None))]
            r2 = 1.0 / (fz[1:] + fz[:-1])
            rise, fall = fc[1:] * fz[1:] * r2 * fy[:-1], -fc[:-1] * fz[:-1] * r2 * fy[1:]
            edge = [a + b for a, b in zip(faces(rise, slice(1, None)), faces(fall, slice(0, -1)))]
            for m, a, b in ((0, flux[0], edge[0]), (comp, flux[1], edge[1])):
                g = a + tn * tw / 6.0 * (b[1:] - b[:-1])
                g = -te * (g[:, 1:] - g[:, :-1])
                inc[m] = inc[m] + (g if ax == 1 else g.transpose(0, 1))
        back = [0, 0, 0]
        for pos, k in enumerate((e2, e1, n)):
            back[2 - k] = pos
        out = out + torch.stack([a.permute(*back) for a in inc])
    return out, max(cfls)


def _net_exact(case, seed):
    """The network, its loss and its gradients by autograd in 64 bits."""
    x, target = _images(case, seed)
    st = _weights(seed)
    w = [torch.tensor(a, dtype=torch.float64, device=_device(), requires_grad=True) for a in st["w"]]
    b = [torch.tensor(a, dtype=torch.float64, device=_device(), requires_grad=True) for a in st["b"]]
    a = x.double().permute(0, 3, 1, 2)
    for k, (cin, cout, act) in enumerate(LAYERS):
        a = torch.nn.functional.conv2d(a, w[k].view(cout, 3, 3, cin).permute(0, 3, 1, 2), b[k], padding=1)
        if act:
            a = torch.nn.functional.gelu(a, approximate="tanh")
    pred = a.permute(0, 2, 3, 1)[..., :4]
    if case["kind"] == "infer":
        return pred.detach()
    d = torch.where(torch.isnan(target), torch.zeros_like(pred), pred - target.double())
    (d * d).sum().div(4 * case["images"] * case["h"] * case["w"]).backward()
    loss = (d * d).sum().detach().reshape(1)
    # the first Adam step moves a weight by lr g / (|g| + eps)
    moved = [(v - 1e-3 * v.grad / (v.grad.abs() + 1e-8)).detach() for v in w]
    return {"loss": loss, "gw": [v.grad for v in w], "gb": [v.grad for v in b], "w": moved}
