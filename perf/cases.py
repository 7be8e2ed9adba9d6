"""Timed workloads of the IB3D hot path, each run through the calls a user's program makes.

A program that uses the library holds a solver context (ib3d_ctx, here `Solver`) with
its fields resident on the GPU and calls the per-step routines on it; the kinds below
are those routines alone and together:

  boundary   velocityBC, solidCellBC, the ghost-point forcing of velocity and pressure
             and drag/lift: the short calls of a step, where launches and latency count
  momentum   the momentum predictor alone (Euler or Adams-Bashforth)
  search     a body put on the grid, searched, moved and re-tagged
  step       whole time steps from a restart state kept on the GPU
  moving     the body moved, re-tagged, then a whole step
  poisson    the pressure-Poisson solve alone, on a clustered cube
  noalloc    the same solve on arrays that the caller owns
  netgrad    loss and gradient of the warm-start network on one batch

Precision: 0 FP64 in the reference's arithmetic, 1 FP32 sweeps in an FP64 defect
correction, 2 FP64 with contracted multiply-adds.
"""
import ctypes
import importlib.util
import json
import math
import pathlib
import sys

import numpy as np
import torch

ROOT = pathlib.Path(__file__).resolve().parent.parent


def _package():
    if "ib3d_gpu_gb300" not in sys.modules:   # the package's folder name is not a Python identifier
        pkg = ROOT / "ib3d-gpu_gb300"
        spec = importlib.util.spec_from_file_location("ib3d_gpu_gb300", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["ib3d_gpu_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["ib3d_gpu_gb300"]


# Solver settings of the headline benchmark's FP32 form.
FAST = dict(precision=1, warm_start=1, criterion=1, inner_sweeps=512, inner_schedule=2, omega_inner=1.9937,
            smooth_sweeps=6, ramp_sweeps=32, max_sweeps=400000)
FAR = ((-5.0, 15.0), (-5.0, 5.0), (-5.0, 5.0))
NEAR = ((-3.0, 6.0), (-3.0, 3.0), (-3.0, 3.0))


def listed():
    return [
        # the smallest grid the smoke test steps on: every call is a few microseconds of work
        dict(name="boundary-40x32x32", kind="boundary", nx=40, ny=32, nz=32, m=8, core=0.75, far=False, sub=3,
             outlet=0),
        # the predictor of the headline benchmark's grid, in the form its steps use
        dict(name="momentum-256x192x192", kind="momentum", nx=256, ny=192, nz=192, m=40, core=0.8, far=True, sub=4,
             precision=1, ab2=False),
        # the bit-exact predictor with the Adams-Bashforth update on a grid of odd extents
        dict(name="momentum-ab2-129x97x75", kind="momentum", nx=129, ny=97, nz=75, m=16, core=0.75, far=True, sub=4,
             precision=0, ab2=True),
        # a body of 5,120 triangles put on the headline grid, then moved by a part of a cell
        dict(name="search-256x192x192", kind="search", nx=256, ny=192, nz=192, m=40, core=0.8, far=True, sub=4),
        # the 96x64x64 sphere in the reference's own arithmetic and stopping test
        dict(name="step-fp64-96x64x64", kind="step", nx=96, ny=64, nz=64, m=16, core=0.75, far=True, sub=4,
             precision=0, re=100.0, omega=1.8, steps=1, net=False, outlet=0, ab2=False),
        # odd extents, convective outlet and Adams-Bashforth: the options of a longer run
        dict(name="step-fp32-129x97x75", kind="step", nx=129, ny=97, nz=75, m=16, core=0.75, far=True, sub=4,
             precision=1, re=150.0, omega=1.95, steps=2, net=False, outlet=1, ab2=True),
        # the headline benchmark: learned warm start (it acts from the second step after a restart)
        dict(name="step-net-256x192x192", kind="step", nx=256, ny=192, nz=192, m=40, core=0.8, far=True, sub=4,
             precision=1, re=275.0, omega=1.99, steps=3, net=True, outlet=0, ab2=False),
        # the moving sphere: the largest grid, whose sweeps do not fit in L2
        dict(name="moving-384x256x256", kind="moving", nx=384, ny=256, nz=256, m=48, core=1.0, far=True, sub=4,
             re=200.0, omega=1.99),
        # the pressure solve alone, as the standalone Poisson benchmark runs it
        dict(name="poisson-fp32-128x128x128", kind="poisson", nx=128, ny=128, nz=128, precision=1, omega=1.85,
             inner=256),
        dict(name="poisson-fast64-100x75x51", kind="poisson", nx=100, ny=75, nz=51, precision=2, omega=1.85, inner=64),
        # a host code that owns its device memory
        dict(name="noalloc-96x64x64", kind="noalloc", nx=96, ny=64, nz=64, omega=1.8, inner=64),
        # one training batch of the warm-start network
        dict(name="netgrad-8x32", kind="netgrad", batch=8, size=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _body_grid(rng, most):
    """Extents between the smallest and `most` x the headline grid's proportions, odd ones among them, the core
    spacing 1/m that leaves room for stretching, and the body's refinement."""
    ny = _log(rng, 32, most)
    nz = max(32, ny + rng.randint(-ny // 5, 0))
    nx = _log(rng, ny, 1.5 * ny) + rng.randint(0, 8)
    m = min(48, 2 * (min(ny, nz) // 8))
    return dict(nx=nx, ny=ny, nz=nz, m=m, core=0.75, far=m >= 14, sub=rng.choice((3, 4, 4)))


def draw(rng):
    kind = rng.choice(("boundary", "momentum", "search", "step", "step", "moving", "poisson", "poisson", "noalloc",
                       "netgrad"))
    if kind == "boundary":
        return dict(kind=kind, **_body_grid(rng, 192), outlet=rng.choice((0, 0, 1)))
    if kind == "momentum":
        return dict(kind=kind, **_body_grid(rng, 192), precision=rng.choice((0, 1, 2)), ab2=rng.random() < 0.3)
    if kind == "search":
        return dict(kind=kind, **_body_grid(rng, 192))
    if kind == "step":
        precision = rng.choice((0, 1, 1, 2))
        return dict(kind=kind, **_body_grid(rng, 72 if precision != 1 else 128), precision=precision,
                    re=round(rng.uniform(80.0, 300.0), 1), omega=round(rng.uniform(1.8, 1.9), 3), steps=rng.choice((1, 2)),
                    net=precision == 1 and rng.random() < 0.3, outlet=rng.choice((0, 0, 1)), ab2=rng.random() < 0.3)
    if kind == "moving":
        return dict(kind=kind, **_body_grid(rng, 112), re=round(rng.uniform(100.0, 250.0), 1),
                    omega=round(rng.uniform(1.85, 1.92), 3))
    if kind == "poisson":
        precision = rng.choice((0, 1, 1, 2))
        most = 144 if precision == 1 else 80
        return dict(kind=kind, nx=_log(rng, 24, most), ny=_log(rng, 24, most), nz=_log(rng, 24, most),
                    precision=precision, omega=round(rng.uniform(1.8, 1.88), 3), inner=rng.choice((64, 128, 256)))
    if kind == "noalloc":
        return dict(kind=kind, nx=_log(rng, 24, 112), ny=_log(rng, 24, 100), nz=_log(rng, 24, 100),
                    omega=round(rng.uniform(1.8, 1.88), 3), inner=rng.choice((16, 32, 64)))
    return dict(kind=kind, batch=rng.randint(1, 8), size=4 * rng.randint(2, 8))


# ------------------------------------------------------------------ what a program has in hand

class _DeviceArray:
    """A field's device memory; it keeps the context that owns the memory alive."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3}


def _field(s, name):
    """A solver field as a torch tensor on the same device memory, (nz+2, ny+2, nx+2) with i fastest."""
    n = s.shape[0] * s.shape[1] * s.shape[2]
    return torch.as_tensor(_DeviceArray(s, s.device_field(name), n), device="cuda").view(s.shape[::-1])


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _workload(case):
    """Grid, body and flow settings (grids.Case) of a case."""
    g = _package().grids
    h = 1.0 / case["m"]
    return g.sphere_case("case", (case["nx"], case["ny"], case["nz"]), h, case["core"], case.get("re", 100.0),
                         min(0.005, 0.08 * h), 1, case.get("omega", 1.95), 1e-6, domain=FAR if case["far"] else NEAR,
                         subdivisions=case["sub"])


def _flow(case, seed, **options):
    """A context on the case's grid with a flow in it: the impulsive start with a seeded 1 % perturbation, and two
    steps of it in the FP32 form, the pressure to a looser tolerance."""
    pkg = _package()
    cs = _workload(case)
    keep = dict(outlet=case.get("outlet", 0), momentum=1 if case.get("ab2") else 0)
    s = pkg.setup_case(cs, **{**FAST, "omega_inner": cs.omega, "eps": 1e-3, **keep})
    u = _field(s, "u")
    s.synchronize()
    u.mul_(1.0 + 0.01 * torch.randn(u.shape, dtype=torch.float64, device="cuda", generator=_generator(seed)))
    torch.cuda.synchronize()
    for n in range(2):
        s.step(n == 0)
    s.set_params(**{"eps": 1e-6, **options})
    s.synchronize()
    return s, cs


STATE = ("u", "v", "w", "ut", "vt", "wt", "p", "pc")


def _restart(s):
    """A restart state kept on the GPU, and what puts it back (ordered with the library's own work)."""
    s.synchronize()
    live = [_field(s, f) for f in STATE]
    saved = [x.clone() for x in live]
    torch.cuda.synchronize()
    return live, saved, torch.cuda.ExternalStream(s.stream())


def _put_back(state):
    with torch.cuda.stream(state["stream"]):
        for x, y in zip(state["live"], state["saved"]):
            x.copy_(y)


def _body(case, seed):
    """The case's sphere, off the grid's centre by a seeded part of a cell."""
    nodes, tris = _package().grids.icosphere(case["sub"], 0.5)
    off = np.random.default_rng(seed).uniform(-0.4, 0.4, 3) / case["m"]
    return nodes + off, tris


def _coefficients(x):
    """(n,3) Poisson coefficients of one axis, Neumann at both ends, and the high end's off-diagonal value."""
    n = len(x) - 1
    d = np.diff(x)
    d = np.concatenate([d[:1], d, d[-1:]])
    r = 0.5 * (d[1:] + d[:-1])                     # spacings of the cell centres, ghost cells included
    lo, hi = r[:n], r[1:n + 1]
    a = np.stack([2.0 / (lo * (lo + hi)), -2.0 / (lo * hi), 2.0 / (hi * (lo + hi))], axis=1)
    last = a[n - 1, 2]
    a[0, 1] += a[0, 0]
    a[n - 1, 1] += a[n - 1, 2]
    a[0, 0] = a[n - 1, 2] = 0.0
    return a, last


def _channel(case):
    """Axes of the clustered box and its coefficients: Neumann faces, and the outlet (high x) at pressure 0."""
    g = _package().grids
    axes = [g.tanh_axis(case[q]) for q in ("nx", "ny", "nz")]
    a = []
    for q, x in enumerate(axes):
        c, last = _coefficients(x)
        if q == 0:
            c[-1, 1] -= 2.0 * last
        a.append(c)
    return axes, a


def _rhs(case, seed):
    """Divergence of a smooth random face velocity (three passes of a box filter), padded, i fastest."""
    axes, _ = _channel(case)
    n = (case["nz"], case["ny"], case["nx"])
    gen = _generator(seed)
    b = torch.zeros([q + 2 for q in n], dtype=torch.float64, device="cuda")
    for dim, x in zip((2, 1, 0), axes):
        v = torch.randn([q + 2 for q in n], dtype=torch.float64, device="cuda", generator=gen)
        for _ in range(3):
            for q in range(3):
                v = (v.roll(1, q) + v + v.roll(-1, q)) / 3.0
        v.select(dim, 0).zero_()
        shape = [1, 1, 1]
        shape[dim] = -1
        d = torch.from_numpy(np.diff(x)).cuda().view(shape)
        inner = [slice(1, -1)] * 3
        low = list(inner)
        low[dim] = slice(0, -2)
        b[1:-1, 1:-1, 1:-1] += (v[tuple(inner)] - v[tuple(low)]) / d
    return b


def _block(case, seed):
    """Flags of a solid ellipsoid in the box, off its centre by a seeded amount."""
    off = np.random.default_rng(seed).uniform(-0.05, 0.05, 3)
    n = (case["nz"], case["ny"], case["nx"])
    c = [torch.linspace(0.0, 1.0, q + 2, dtype=torch.float64, device="cuda") - 0.5 - off[k] for k, q in enumerate(n)]
    r = c[0].view(-1, 1, 1) ** 2 + c[1].view(1, -1, 1) ** 2 + c[2].view(1, 1, -1) ** 2
    return (r < 0.12 ** 2).to(torch.uint8)


def _batch(case, seed):
    """Inputs of unit scale and targets of the size that the network is trained on, smooth in space."""
    gen = _generator(seed)
    B, S = case["batch"], case["size"]
    x = torch.randn(B, 5, S, S, S, generator=gen, device="cuda")
    for dim in (2, 3, 4):
        x = (x.roll(1, dim) + 2.0 * x + x.roll(-1, dim)) / 2.45
    x = x.cpu().numpy()
    return np.ascontiguousarray(x[:, :4].transpose(0, 2, 3, 4, 1)), np.ascontiguousarray(0.3 * x[:, 4])


def _weights():
    folder = ROOT / "ib3d-gpu_gb300" / "weights"
    info = json.loads((folder / "networks.json").read_text())
    return np.fromfile(folder / info["default"], dtype="<f4"), int(info["networks"][info["default"]]["coarsen"])


def _network():
    net = _package().Net(seed=0)
    w, coarsen = _weights()
    net.set_coarsening(coarsen)
    net.set_params(w)
    return net


def prepare(case, seed):
    kind, pkg = case["kind"], _package()
    if kind == "boundary":
        s, _ = _flow(case, seed)
        s.stress(True)
        return dict(case=case, s=s, out=[_field(s, f) for f in ("ut", "vt", "wt", "p")])
    if kind == "momentum":
        s, _ = _flow(case, seed, precision=case["precision"])
        return dict(case=case, s=s, out=[_field(s, f) for f in ("ut", "vt", "wt")])
    if kind == "search":
        cs = _workload(case)
        s = pkg.Solver(cs.x, cs.y, cs.z, pkg.default_params(re=cs.re, deltat=cs.dt))
        return dict(case=case, s=s, cs=cs, body=_body(case, seed))
    if kind == "step":
        plain = dict(precision=case["precision"], warm_start=0, criterion=0)
        s, _ = _flow(case, seed, **({} if case["precision"] == 1 else plain))
        net = None
        if case["net"]:
            net = _network()
            s.set_params(warm_start=2, **({"omega_inner": 1.9937} if case["omega"] > 1.95 else {}))
        live, saved, stream = _restart(s)
        return dict(case=case, s=s, net=net, live=live, saved=saved, stream=stream)
    if kind == "moving":
        s, cs = _flow(case, seed)
        if case["omega"] > 1.95:
            s.set_params(omega_inner=1.9937)
        nodes, tris = _body(case, seed)
        s.set_mesh(nodes, tris)
        s.move_body(0.0, 0.0, 0.0, 0.0, 0.2, 0.0)
        live, saved, stream = _restart(s)
        return dict(case=case, s=s, cs=cs, body=(nodes, tris), live=live, saved=saved, stream=stream)
    if kind == "poisson":
        axes, a = _channel(case)
        p = pkg.default_params(re=100.0, deltat=1.0, omega=case["omega"], eps=1e-8, max_sweeps=200000, criterion=1,
                               precision=case["precision"], check_every=8, inner_sweeps=case["inner"])
        s = pkg.Solver(*axes, p)
        s.set_poisson_coefficients(*a)
        _field(s, "b").copy_(_rhs(case, seed))
        torch.cuda.synchronize()
        return dict(case=case, s=s, out=_field(s, "pc"))
    if kind == "noalloc":
        _, a = _channel(case)
        coef = [torch.from_numpy(np.ascontiguousarray(c.T)).cuda() for c in a]
        b = _rhs(case, seed)
        return dict(case=case, coef=coef, cell=_block(case, seed), b=b, pc=torch.zeros_like(b),
                    sweeps=np.zeros(1, np.int64), residual=np.zeros(1))
    if kind == "netgrad":
        x, t = _batch(case, seed)
        return dict(case=case, net=_network(), x=x, t=t)
    raise KeyError(kind)


# ------------------------------------------------------------------ one pass

def _placed(state, step=0.2):
    """The body put at its first position and searched, then moved by a fifth of a cell along y and re-tagged."""
    s, cs = state["s"], state["cs"]
    s.set_mesh(*state["body"])
    s.search(cs.box)
    s.move_body(0.0, step / state["case"]["m"], 0.0, 0.0, 0.2, 0.0)
    return s.selective_retag()


def _ib_room(case):
    """Room for the IB cells, as a caller that does not know their number yet sets aside (the unit sphere's surface
    cuts about 4.7 m^2 cells)."""
    return 8 * case["m"] ** 2 + 512


def run(state):
    case = state["case"]
    kind, s = case["kind"], state.get("s")
    if kind == "boundary":
        s.velocity_bc()
        s.solid_cell_bc()
        s.velocity_forcing()
        s.velocity_bc()
        s.pressure_forcing()
        if case["outlet"]:
            s.calculate_uc()
        return state["out"] + [s.stress(False)]
    if kind == "momentum":
        (s.ns_momentum_ab if case["ab2"] else s.ns_momentum)()
        return state["out"]
    if kind == "search":
        counts = _placed(state)
        n, room = counts["ib"], _ib_room(case)
        ib, nelp, nd = np.zeros(3 * room, np.int64), np.zeros(room, np.int64), np.zeros(7 * room)
        i64, f64 = ctypes.POINTER(ctypes.c_int64), ctypes.POINTER(ctypes.c_double)
        rc = s.L.ib3d_get_search(s._h, None, ib.ctypes.data_as(i64), nelp.ctypes.data_as(i64), nd.ctypes.data_as(f64))
        if rc:
            raise RuntimeError("ib3d_get_search: %d" % rc)
        return {"counts": np.array([counts[q] for q in ("fluid", "solid", "ib", "red", "black")]), "ib": ib,
                "nelp": nelp, "normdis": nd}
    if kind == "step":
        _put_back(state)
        if state["net"] is not None:
            s.attach_net(state["net"])          # a restart begins without the previous pressures
        coefs = [s.step(False)[1] for _ in range(case["steps"])]
        return state["live"] + [np.array(coefs)]
    if kind == "moving":
        _put_back(state)
        _placed(state)
        return state["live"] + [s.step(True)[1]]
    if kind == "poisson":
        s.redblack_sor()
        return state["out"]
    if kind == "noalloc":
        state["pc"].zero_()
        c, i64 = state["coef"], ctypes.POINTER(ctypes.c_int64)
        rc = _package().lib().ib3d_pressure_solve_noalloc(
            case["nx"], case["ny"], case["nz"], c[0].data_ptr(), c[1].data_ptr(), c[2].data_ptr(),
            state["cell"].data_ptr(), state["b"].data_ptr(), 1.0, state["pc"].data_ptr(), case["omega"], 1e-8, 200000,
            case["inner"], torch.cuda.current_stream().cuda_stream, state["sweeps"].ctypes.data_as(i64),
            state["residual"].ctypes.data_as(ctypes.POINTER(ctypes.c_double)))
        if rc:
            raise RuntimeError("ib3d_pressure_solve_noalloc: %d" % rc)
        return state["pc"]
    loss, grad, out = state["net"].loss_grad(state["x"], state["t"])
    return {"loss": loss, "grad": grad, "out": out}


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """Every array read or written once, and the arithmetic of the reference's formulas; an iterative solve's with
    the sweeps that red-black over-relaxation takes on such a grid (about 10 per cell of the longest edge)."""
    kind = case["kind"]
    if kind == "netgrad":
        M = case["batch"] * case["size"] ** 3
        pairs = 16 * 16 * 3 + 48 * 16 + (16 * 32 + 32 * 32 * 2 + 96 * 32) / 8 + (32 * 64 + 64 * 64) / 64
        return {"bytes": M * 4 * 6 + 359761 * 8, "flops": 3 * 2 * 27 * M * pairs}
    cells = case["nx"] * case["ny"] * case["nz"]
    sweeps = 10 * max(case["nx"], case["ny"], case["nz"])
    faces = 2 * (case["nx"] * case["ny"] + case["ny"] * case["nz"] + case["nx"] * case["nz"])
    tri = 20 * 4 ** case.get("sub", 0)
    ib = 12.0 * case.get("m", 0) ** 2 / 4 * math.pi / 3      # cells that the unit sphere's surface cuts
    if kind == "boundary":
        return {"bytes": cells + 8 * 4 * faces + 7 * ib * 9 * 8 + tri * 41 * 8, "flops": 7 * ib * 100 + tri * 500}
    if kind == "momentum":
        return {"bytes": cells * (57 + (48 if case["ab2"] else 0)), "flops": 230.0 * cells}
    if kind == "search":
        box = (2 * (0.5 * case["m"] + 4)) ** 3
        return {"bytes": 2 * (cells + tri * 9 * 8 + ib * 100), "flops": 2 * 9.0 * box * math.log2(tri)}
    if kind == "poisson":
        return {"bytes": 16.0 * cells, "flops": 15.0 * cells * sweeps}
    if kind == "noalloc":
        return {"bytes": 17.0 * cells, "flops": 15.0 * cells * sweeps}
    n = case.get("steps", 1)
    return {"bytes": n * 113.0 * cells, "flops": n * cells * (250.0 + 15.0 * sweeps)}


# ------------------------------------------------------------------ the same in 64 bits

def exact(case, seed):
    kind = case["kind"]
    if kind == "momentum":
        return None if case["ab2"] else _exact_momentum(case, seed)   # the previous residual is the context's own
    if kind == "search":
        return _exact_search(case, seed)
    if kind == "poisson":
        return _exact_pressure(case, _rhs(case, seed), None)
    if kind == "noalloc":
        return _exact_pressure(case, _rhs(case, seed), _block(case, seed))
    if kind == "netgrad":
        return _exact_netgrad(case, seed)
    return None     # whole steps, and the forcing, whose ghost values depend on one another in the serial order


def _exact_pressure(case, b, cell):
    """The solution of the seven-point system: conjugate gradients on the row-scaled, symmetric form, to rounding."""
    _, a = _channel(case)
    axes = _channel(case)[0]
    shape = ((1, 1, -1), (1, -1, 1), (-1, 1, 1))
    w = 1.0
    off, diag = [], 0.0
    fluid = torch.ones_like(b[1:-1, 1:-1, 1:-1]) if cell is None else (cell[1:-1, 1:-1, 1:-1] == 0).double()
    for q in range(3):
        d = np.diff(axes[q])
        d = np.concatenate([d[:1], d, d[-1:]])
        wq = 0.5 * (0.5 * (d[1:-1] + d[:-2]) + 0.5 * (d[2:] + d[1:-1]))      # makes the axis' operator symmetric
        w = w * torch.from_numpy(wq).cuda().view(shape[q])
        c = [torch.from_numpy(np.ascontiguousarray(a[q][:, k])).cuda().view(shape[q]) for k in range(3)]
        off.append((c[0], c[2]))
        diag = diag + c[1]

    def apply(x):
        p = torch.zeros_like(b)
        p[1:-1, 1:-1, 1:-1] = x
        y = diag * x
        y = y + off[0][0] * p[1:-1, 1:-1, :-2] + off[0][1] * p[1:-1, 1:-1, 2:]
        y = y + off[1][0] * p[1:-1, :-2, 1:-1] + off[1][1] * p[1:-1, 2:, 1:-1]
        y = y + off[2][0] * p[:-2, 1:-1, 1:-1] + off[2][1] * p[2:, 1:-1, 1:-1]
        return -w * y * fluid

    r = -w * b[1:-1, 1:-1, 1:-1] * fluid
    scale = -w * diag
    x = torch.zeros_like(r)
    z = r / scale
    p, rz, first = z.clone(), (r * z).sum(), (r * r).sum()
    for n in range(6000):
        q = apply(p)
        alpha = rz / (p * q).sum()
        x += alpha * p
        r -= alpha * q
        z = r / scale
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
        if n % 50 == 49 and (r * r).sum() <= 1e-28 * first:
            break
    out = torch.zeros_like(b)
    out[1:-1, 1:-1, 1:-1] = x
    return out


def _station(t1, t2, t3):
    """The twelve coefficients of the third-order upwind stencil at one station, from its three spacing ratios."""
    f1, f2, f3 = t3, 2 * t3 + t3 ** 2, 3 * t3 + 3 * t3 ** 2 + t3 ** 3
    f4 = 4 * t3 + 6 * t3 ** 2 + 4 * t3 ** 3 + t3 ** 4
    f5, f6 = 1 / (t1 * t2), (2 * t1 + 1) / (t1 * t2) ** 2
    f7 = (3 * t1 ** 2 + 3 * t1 + 1) / (t1 * t2) ** 3
    f8 = (4 * t1 ** 3 + 6 * t1 ** 2 + 4 * t1 + 1) / (t1 * t2) ** 4
    i4 = 1 / t2 ** 4
    s55, s56, s57 = -(f1 * i4 + f4 / t2), f4 / t2 ** 2 - f2 * i4, -(f3 * i4 + f4 / t2 ** 3)
    s65, s66, s67 = f5 + f8, f8 - f6, f7 + f8
    s74, s75, s76 = f4 - f1, f4 - f2, f4 - f3
    s84, s85, s86 = f5 * i4 - f8 / t2, f8 / t2 ** 2 - f6 * i4, f7 * i4 - f8 / t2 ** 3
    s91, s92, s93 = s66 * i4, -s56, -(-i4 * s66 + s56 * f8)
    s94, s95 = -s56 + s66 * f4, s56 * f8 - s66 * f4
    s96, s97 = s56 * s65 - s66 * s55, s56 * s67 - s66 * s57
    s101, s102, s103, s104 = s85, -s85 * (1 + f4), -s75 * i4, s75 * (f8 + i4)
    s105, s106, s107 = s75 * f8 - s85 * f4, s75 * s84 - s85 * s74, s75 * s86 - s85 * s76
    low = [s97 * s101 - s107 * s91, s97 * s102 + s107 * s93, s95 * s107 - s105 * s97, s94 * s107 + s104 * s97,
           s97 * s103 - s107 * s92, s97 * s106 - s107 * s96]
    g = t3 + t3 ** 2
    high = [1 + t1, -(1 + t1) * (1 + t3) ** 2, (1 + 2 * t1) * g * t2 + (1 + t1) * (2 * t3 + t3 ** 2),
            -(1 + t1) ** 2 * g * t2, t1 ** 2 * t2 * g, (1 + t1) * g * t2]
    return low + high


def _exact_momentum(case, seed):
    """The predictor on the same flow: convection (third-order upwind away from walls and the body, else first-order),
    diffusion and the pressure gradient."""
    s, cs = _flow(case, seed, precision=case["precision"])
    V = [_field(s, f).clone() for f in "uvw"]
    p = _field(s, "p").clone()
    T = [_field(s, f).clone() for f in ("ut", "vt", "wt")]
    torch.cuda.synchronize()
    cell = torch.from_numpy(np.ascontiguousarray(s.get_search()["cell"].transpose(2, 1, 0))).cuda()
    s.close()
    n = (case["nx"], case["ny"], case["nz"])
    dims, shape = (2, 1, 0), ((1, 1, -1), (1, -1, 1), (-1, 1, 1))
    at = lambda t, a, k: t.roll(-k, dims[a])                  # the value k cells further along axis a
    ix = [torch.arange(1, q + 3, device="cuda").view(sh) for q, sh in zip(n, shape)]
    own, half = [], []
    for a, x in enumerate((cs.x, cs.y, cs.z)):
        d = np.diff(x)
        d = np.concatenate([d[:1], d, d[-1:]])                # d[m-1]: spacing of cell m = 1..n+2
        m = np.arange(2, n[a] + 2)
        dm, dp, dl = d[m - 1], d[m], d[m - 2]
        own_t, half_t = np.ones((12, n[a] + 2)), np.ones((12, n[a] + 2))
        k = np.arange(2, n[a] + 1)
        d0, d1, d2, d3 = d[k - 2], d[k - 1], d[k], d[k + 1]
        own_t[:, k - 1] = _station(d1 / d0, d2 / d1, d3 / d2)
        h1 = np.where(k == 2, d0, 0.5 * (d0 + d[np.maximum(k - 3, 0)]))
        h2, h3, h4 = 0.5 * (d1 + d0), 0.5 * (d1 + d2), 0.5 * (d2 + d3)
        half_t[:, k - 1] = _station(h2 / h1, h3 / h2, h4 / h3)
        put = lambda v: torch.from_numpy(np.concatenate([[1.0], v, [1.0]])).cuda().view(shape[a])
        own.append((put(dp), put(dm), [torch.from_numpy(v.copy()).cuda().view(shape[a]) for v in own_t]))
        half.append((put(0.5 * (dm + dp)), put(0.5 * (dm + dl)),
                     [torch.from_numpy(v.copy()).cuda().view(shape[a]) for v in half_t]))
    fluid = cell == 0
    for a in range(3):
        fluid = fluid & (ix[a] >= 2) & (ix[a] <= n[a] + 1)
    clear = torch.ones_like(fluid)
    for a in range(3):
        clear = clear & (at(cell, a, 1) != 2) & (at(cell, a, -1) != 2)
    out = []
    for c in range(3):
        q0, total = V[c], 0.0
        inner = clear.clone()
        for a in range(3):
            inner = inner & (ix[a] != 2) & (ix[a] < (n[a] if a == c else n[a] + 1))
        for a in range(3):
            hi, lo, k = own[a] if a == c else half[a]
            qp, qm = at(q0, a, 1), at(q0, a, -1)
            if a == c:
                adv = q0
            else:
                wgt = own[c][0] / (own[c][0] + own[c][1])
                face = lambda t: at(t, c, 1) + wgt * (t - at(t, c, 1))
                adv = 0.5 * (face(V[a]) + face(at(V[a], a, -1)))
            five = [at(q0, a, 2), qp, q0, qm, at(q0, a, -2)]
            third = (adv * sum(x * y for x, y in zip(k[:5], five)) / (k[5] * hi)
                     + adv.abs() * sum(x * y for x, y in zip(k[6:11], five)) / (2.0 * k[11] * lo))
            r = lo / hi
            first = (adv / hi * (-qm / (r * (r + 1)) - (1 - 1 / r) * q0 + r / (r + 1) * qp)
                     - adv.abs() / (2 * hi) * (2 * qm / (r * (r + 1)) - 2 * q0 / r + 2 * qp / (r + 1)))
            total = total - torch.where(inner, third, first)
            span = (hi + lo)
            total = total + 2.0 / span * ((qp - q0) / hi + (qm - q0) / lo) / cs.re
        grad = (p - at(p, c, 1)) / half[c][0]
        out.append(torch.where(fluid, q0 + cs.dt * (total + grad), T[c]))
    return out


def _exact_search(case, seed):
    """Nearest centroid of each cell of the box after the move, its flag, and the IB cells' normal distances."""
    cs = _workload(case)
    nodes, tris = _body(case, seed)
    P = torch.from_numpy(nodes + np.array([0.0, 0.2 / case["m"], 0.0])).cuda()[torch.from_numpy(tris - 1).cuda()]
    centre = P.sum(1) / 3.0
    nrm = torch.linalg.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    lo, hi = [], []
    for a, x in enumerate((cs.x, cs.y, cs.z)):
        i = np.arange(cs.box[2 * a], cs.box[2 * a + 1] + 1)
        lo.append(torch.from_numpy(x[i - 2]).cuda())
        hi.append(torch.from_numpy(x[i - 1]).cuda())
    grid = lambda v: torch.stack([t.permute(2, 1, 0).reshape(-1) for t in torch.meshgrid(*v, indexing="ij")], 1)
    L, H = grid(lo), grid(hi)
    mid = 0.5 * (L + H)
    near = torch.cat([((m[:, None, :] - centre[None]) ** 2).sum(2).argmin(1) for m in mid.split(8192)])
    dot = lambda x: ((x - centre[near]) * nrm[near]).sum(1)
    corners = torch.stack([dot(torch.stack([(H if q >> a & 1 else L)[:, a] for a in range(3)], 1)) for q in range(8)])
    cut = ~((corners <= -1e-16).all(0) | (corners > -1e-16).all(0))
    at = [dot(mid)]
    for a in range(3):
        for side in (L, H):
            x = mid.clone()
            x[:, a] = side[:, a]
            at.append(dot(x))
    nd = torch.zeros(7 * _ib_room(case), dtype=torch.float64)
    found = torch.cat([t[cut] for t in at]).cpu()             # seven blocks, one per distance
    nd[:len(found)] = found
    return {"counts": None, "ib": None, "nelp": None, "normdis": nd}


def _exact_netgrad(case, seed):
    """The network's loss, gradient and output without any rounding to 16 bits."""
    import torch.nn.functional as F
    x, t = _batch(case, seed)
    out_ch, in_ch = (16, 16, 32, 32, 64, 64, 32, 32, 16, 16), (16, 16, 16, 32, 32, 64, 96, 32, 48, 16)
    p = torch.from_numpy(_weights()[0]).double().cuda().requires_grad_()
    x = F.pad(torch.from_numpy(x).double().cuda().permute(0, 4, 1, 2, 3), (0, 0, 0, 0, 0, 0, 0, 12))
    at, layers = 0, []
    for n, k in zip(out_ch, in_ch):
        layers.append((p[at:at + n * 27 * k].view(n, 27, k).permute(0, 2, 1).reshape(n, k, 3, 3, 3),
                       p[at + n * 27 * k:at + n * 27 * k + n]))
        at = (at + n * 27 * k + n + 7) // 8 * 8

    def conv(v, l):
        """A 3x3x3 convolution as 27 products of matrices: cuDNN has no quick one in 64 bits."""
        w, b = layers[l]
        D, Hh, W = v.shape[2:]
        v = F.pad(v, (1, 1, 1, 1, 1, 1))
        y = b.view(1, -1, 1, 1, 1)
        for q in range(27):
            z, r, c = q // 9, q // 3 % 3, q % 3
            y = y + torch.einsum("bkzyx,nk->bnzyx", v[:, :, z:z + D, r:r + Hh, c:c + W], w[:, :, z, r, c])
        return F.relu(y)

    up = lambda v: F.interpolate(v, scale_factor=2, mode="nearest")
    e1 = conv(conv(x, 0), 1)
    e2 = conv(conv(F.avg_pool3d(e1, 2), 2), 3)
    mid = conv(conv(F.avg_pool3d(e2, 2), 4), 5)
    d2 = conv(conv(torch.cat([up(mid), e2], 1), 6), 7)
    d1 = conv(conv(torch.cat([up(d2), e1], 1), 8), 9)
    y = torch.einsum("bkzyx,k->bzyx", d1, p[at:at + 16]) + p[at + 16]
    loss = ((y - torch.from_numpy(t).double().cuda()) ** 2).mean()
    loss.backward()
    return {"loss": loss.detach(), "grad": p.grad, "out": y.detach()}
