"""Performance cases of the time-step library: what a user's program has it do, through the Python
binding's public calls, over the range of sizes and options in use.

Kinds of case (``case["kind"]``):

* ``stokes``   the first solve of a run: the restart's v, P are uploaded, ``runtime.time_step`` runs
               with only the mechanics switched on, v and P come back as the restart file keeps them;
* ``heat``     ``steps`` time steps with only the heat equation switched on (implicit solve and the
               markers' temperature update), then the temperatures of nodes and markers come back;
* ``markers``  ``steps`` kinematic time steps: markers carried by the velocity at hand (RK4 and
               rheology), then marker -> node averages; markers and nodal fields come back;
* ``step``     a whole run segment between two output files: the restart goes up, ``steps`` full time
               steps (Stokes, heat, markers, nodes), the state comes down;
* ``unet``     the learned warm start's network on one sample: its output, or output, loss and
               parameter gradients.

Models: ``sphere`` (a dense stiff sphere in a Newtonian box), ``plastic`` (the same below a
Drucker-Prager matrix) and ``inclusions`` (spheres in an Arrhenius matrix, viscosities clamped to
1e19 .. 1e22 Pa s like the subduction model's mantle), with 2 x 2 x 2 or 3 x 3 x 3 jittered markers per cell.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from i3elvis_b200 import abi, config, lib, model, runtime
from i3elvis_b200.prn import YEAR, Prn
from i3elvis_b200.warmstart import UNet

RGAS = 8.314
T_TOP, T_BOTTOM = 273.0, 1573.0
NODES = ("ro", "nu", "nxx", "nxy", "nxz", "nyz", "tk", "cp", "kt")
FLOW = ("pr", "vx", "vy", "vz")
MOVED = ("markx", "marky", "markz", "markk", "markv", "marke", "markft", "markt")


def listed():
    def c(name, kind, shape, **kw):
        return dict(name=name, kind=kind, nx=shape[0], ny=shape[1], nz=shape[2], **kw)
    cube = lambda n: (n, n, n)  # noqa: E731
    mixed = dict(precision=1, krylov=8)
    return [
        # the smallest model anyone solves (tests, tutorials): every launch is latency
        c("stokes 17 mixed", "stokes", cube(17), model="sphere", mnum=2, **mixed),
        # the CPU-sized benchmark model with the library's default solver (FP64 multigrid)
        c("stokes 33 fp64", "stokes", cube(33), model="sphere", mnum=3, precision=0, krylov=0),
        # a box with three different sides and the Arrhenius law's viscosity contrast
        c("stokes 61x37x53 mixed", "stokes", (61, 37, 53), model="inclusions", mnum=2, **mixed),
        # the benchmark's half-size grid
        c("stokes 65 mixed", "stokes", cube(65), model="inclusions", mnum=2, **mixed),
        # the benchmark's grid, cold start
        c("stokes 129 mixed", "stokes", cube(129), model="inclusions", mnum=2, **mixed),
        # heat steps at the half size with the benchmark's 27 markers per cell
        c("heat 65", "heat", cube(65), model="inclusions", mnum=3, steps=4, marker_exact=0),
        # heat steps on the benchmark's grid
        c("heat 129", "heat", cube(129), model="inclusions", mnum=2, steps=4, marker_exact=0),
        # small yielding model, marker arithmetic in the reference's operation order
        c("markers 33 plastic exact", "markers", cube(33), model="plastic", mnum=3, steps=8, marker_exact=1),
        # a box of three different sides with the benchmark's markers per cell (12 M), default arithmetic
        c("markers 97x65x77", "markers", (97, 65, 77), model="inclusions", mnum=3, steps=8, marker_exact=0),
        # a whole run segment of the small benchmark model
        c("step 33", "step", cube(33), model="sphere", mnum=3, steps=4, marker_exact=0, warm_start=3, **mixed),
        # a whole run segment on the benchmark's grid
        c("step 129", "step", cube(129), model="inclusions", mnum=2, steps=3, marker_exact=0, warm_start=3, **mixed),
        # one training sample of the learned warm start at its training size: forward and backward
        c("unet gradients 33", "unet", cube(33), grads=True),
    ]


def _odd(rng, lo, hi):
    """An odd number of nodes, log-uniform: the level rule halves the inner nodes."""
    return 2 * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2)) + 1


def draw(rng):
    kind = rng.choice(("stokes", "stokes", "heat", "markers", "step", "unet"))
    if kind == "unet":
        # every axis needs n - 1 divisible by 8
        nx, ny, nz = (8 * rng.randint(2, 8) + 1 for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, grads=rng.random() < 0.5)
    top = {"stokes": 120, "heat": 120, "markers": 76, "step": 100}[kind]
    n = _odd(rng, 16, top)
    if kind in ("stokes", "step"):
        # small models are spheres, larger ones inclusions; sides up to a factor of 1.5 apart
        least = 15 if n <= 41 else 37
        dims = [n, max(least, _odd(rng, n / 1.5, n)), max(least, _odd(rng, n / 1.5, n))]
    else:
        dims = [n, max(15, _odd(rng, n / 2, n)), max(15, _odd(rng, n / 2, n))]
    rng.shuffle(dims)
    c = dict(kind=kind, nx=dims[0], ny=dims[1], nz=dims[2], mnum=rng.choice((2, 3)), model="sphere" if n <= 41 else "inclusions")
    if kind in ("heat", "markers"):
        c.update(steps=rng.randint(2, 6), marker_exact=rng.choice((0, 0, 1)))
        if kind == "markers" and rng.random() < 0.3:
            c["model"] = "plastic"
    else:
        c.update(precision=1, krylov=8)
        if kind == "stokes" and c["model"] == "sphere" and rng.random() < 0.5:
            c.update(precision=0, krylov=0)
        if kind == "step":
            c.update(steps=rng.randint(1, 3), marker_exact=0, warm_start=3)
    return c


# ---------------------------------------------------------------------------------------
# models
# ---------------------------------------------------------------------------------------
def _levels(case):
    """Coarse levels of the benchmark's configurations: 2 at 33 nodes, 3 at 65, 4 at 129."""
    n = min(case["nx"], case["ny"], case["nz"])
    return 2 if n < 37 else 3 if n < 100 else 4


def _sweeps(case, levels):
    """The benchmark's relaxation sweeps: light ones when the V-cycle preconditions FGMRES, the
    reference's proportions otherwise."""
    if case.get("krylov"):
        light = (2, 4, 4, 8)[:levels]
        return light + (0,), light + (4,)
    heavy = (8, 16, 16, 32)[:levels]
    return heavy + (0,), heavy + (64,)


def _size(case):
    """Box size in metres: 100 km (spheres) or 200 km along the longest side, cubic cells."""
    dims = case["nx"], case["ny"], case["nz"]
    h = (200e3 if case["model"] == "inclusions" else 100e3) / (max(dims) - 1)
    return tuple(h * (n - 1) for n in dims), h


def _bodies(case, seed):
    """Seeded spheres (rock type, centre, radius) and the rock table."""
    rng = np.random.default_rng(seed)
    size, h = _size(case)
    size = np.array(size)
    if case["model"] != "inclusions":
        mat = model.Rock(nu=1e21, ro=3300.0)
        centre, rho = size * rng.uniform(0.4, 0.6, 3), 3400.0
        if case["model"] == "plastic":
            mat = dataclasses.replace(mat, a0=1e7, a1=1e7, b0=0.6, b1=0.6)
            centre[1], rho = 0.3 * size[1], 4300.0
        rocks = {model.MATRIX: mat, model.SPHERE: model.Rock(nu=1e23, ro=rho)}
        return [(model.SPHERE, centre, 0.2 * size.min())], rocks
    count = 100 if max(case["nx"], case["ny"], case["nz"]) > 50 else 30
    eta, energy, t_ref = 1e21, 5e5, 923.0
    mat = model.Rock(nu=eta / math.exp(energy / (RGAS * t_ref)), dh=energy, n0=1e19, n1=1e22, ro=3300.0)
    types = model.INCLUSION_TYPES
    rocks = {model.MATRIX: mat}
    for b, t in enumerate(types):
        rocks[t] = dataclasses.replace(mat, ro=3250.0 + 200.0 * (b + 0.5) / len(types))
    bodies = [(types[int(rng.integers(len(types)))], size * rng.uniform(0.1, 0.9, 3), h * rng.uniform(1.3, 5.1))
              for _ in range(count)]
    return bodies, rocks


def _markers(case, seed):
    """Markers on a jittered sub-grid of every cell in the reference's order, on the GPU: positions,
    rock types and temperatures (FP32, as the restart file holds them)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    size, h = _size(case)
    m = case["mnum"]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    view = {0: (1, nx - 1, 1, 1, m, 1), 1: (1, 1, ny - 1, 1, 1, m), 2: (nz - 1, 1, 1, m, 1, 1)}
    full = (nz - 1, nx - 1, ny - 1, m, m, m)
    pos = []
    for axis, n in ((0, nx), (1, ny), (2, nz)):
        at = (torch.arange((n - 1) * m, device="cuda", dtype=torch.float64) + 0.5) * (h / m)
        at = at.reshape(view[axis]).expand(full).reshape(-1)
        r = torch.randint(-100, 101, at.shape, generator=g, device="cuda", dtype=torch.int16)
        pos.append((at + r.to(torch.float64) * (0.5 * h / m / 100)).float())
    bodies, rocks = _bodies(case, seed)
    types = torch.full_like(pos[0], model.MATRIX, dtype=torch.int8)
    hot = torch.zeros_like(pos[0])
    for rock, c, r in bodies:
        inside = sum((p - float(x)) ** 2 for p, x in zip(pos, c)) <= float(r) ** 2
        types.masked_fill_(inside, rock)
        hot.masked_fill_(inside, 120.0)
    temp = T_TOP + (T_BOTTOM - T_TOP) * pos[1] / size[1]
    if case["kind"] in ("heat", "markers"):
        # something to diffuse and to carry: a broad swell and warm bodies
        temp = temp + 60.0 * torch.sin(math.pi * pos[1] / size[1]) * torch.cos(2 * math.pi * pos[0] / size[0]) + hot
    return pos, types, temp.float(), rocks


@functools.lru_cache(maxsize=None)
def _grid(nx, ny, nz, mnum, levels, size):
    """Grid lines, boundary rows and an empty image of a model of this shape."""
    spec = model.ModelSpec(shape=(nx, ny, nz), size=size, mnum=(mnum,) * 3, multinum=levels, t_top=T_TOP, t_bottom=T_BOTTOM)
    one = np.zeros(1, np.float32)
    rocks = {t: model.Rock() for t in (model.MATRIX, max(model.INCLUSION_TYPES))}
    return model.make_prn(spec, rocks, np.full(1, model.MATRIX, np.int8), (one, one, one))


def _image(case, seed):
    """The restart image a run begins with: grid, boundary rows, rock table, markers."""
    base = _grid(case["nx"], case["ny"], case["nz"], case["mnum"], _levels(case), _size(case)[0])
    (x, y, z), types, temp, rocks = _markers(case, seed)
    table = {f: np.zeros_like(v) for f, v in base.rocks.items()}
    for t, r in rocks.items():
        for f in table:
            table[f][t] = getattr(r, f)
    n = x.numel()
    marks = {f: np.broadcast_to(np.float32(0), n) for f in ("w", "d", "v", "e", "ex", "ft", "rr", "rn")}
    marks.update(x=x.cpu().numpy(), y=y.cpu().numpy(), z=z.cpu().numpy(), k=temp.cpu().numpy(), t=types.cpu().numpy())
    return Prn(dict(base.head, marknum=n), table, base.nodes, base.gx, base.gy, base.gz, base.bond, marks)


def _time_step(case):
    """Seconds of a prescribed time step: half a cell at the kinematic flow's 1 nm/s, a tenth of a cell's
    diffusion time for heat alone."""
    h = _size(case)[1]
    return 0.5 * h / 1e-9 if case["kind"] == "markers" else 0.3 * h * h / 1e-6


def _mode(case):
    levels = _levels(case)
    down, up = _sweeps(case, levels)
    kind = case["kind"]
    plan = config.OutFile("out.prn", cyc0max=case.get("steps", 1), maxxystep=0.5 * _size(case)[1], nubeg=1e18, nuend=1e24,
                          maxtmstep_yr=1e9 if kind in ("stokes", "step") else _time_step(case) / YEAR,
                          p0koef=0.71, p1koef=1.0, p0koef2=0.71, p1koef2=0.0, multinum=levels, multinum2=levels)
    return config.Mode(multinum=levels, multicyc=1, multinnn=(down, up), p0koef=0.71, p1koef=1.0, v0koef=0.7, v1koef=0.7,
                       nubeg=1e18, nuend=1e24, files=[plan], movemod=int(kind in ("stokes", "step")),
                       tempmod=int(kind in ("heat", "step")), markmod=2 if kind in ("markers", "step") else 0,
                       gridmod=int(kind in ("markers", "step")))


def _roll(case):
    """A divergence-free convection roll in x-y and z-y (1 nm/s, no flow through the walls), each component
    at its own staggered points."""
    (lx, ly, lz), h = _size(case)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    at = lambda n, mid: (np.arange(n) + (0.5 if mid else 0.0)) * h  # noqa: E731
    u, w = 1e-9, 0.5e-9

    def field(f, mx, my, mz):
        z, x, y = at(nz, mz)[:, None, None] / lz, at(nx, mx)[None, :, None] / lx, at(ny, my)[None, None, :] / ly
        return np.broadcast_to(f(math.pi * x, math.pi * y, math.pi * z), (nz, nx, ny)).astype(np.float32).reshape(-1)
    vx = field(lambda x, y, z: u * np.sin(x) * np.cos(y) + 0 * z, False, True, True)
    vz = field(lambda x, y, z: w * np.sin(z) * np.cos(y) + 0 * x, True, True, False)
    vy = field(lambda x, y, z: -(u * ly / lx * np.cos(x) + w * ly / lz * np.cos(z)) * np.sin(y), True, False, True)
    return vx, vy, vz


def _part(m, keep, arrays):
    """A model description that names only the arrays to be copied (a null pointer is skipped)."""
    p = abi.Model.from_buffer_copy(m)
    for f, kind in abi.Model._fields_:
        if f in FLOW + abi.NODE_F32 + abi.STRESS_F32 + abi.MARK_F32 + ("markt",):
            setattr(p, f, arrays[f].ctypes.data_as(kind) if f in keep else kind())
    return p


def _pinned(n, dtype):
    return torch.empty(n, dtype=dtype, pin_memory=True).numpy()


def _space(names, nodes, marks):
    """Page-locked arrays for a download."""
    size = lambda f: marks if f.startswith("mark") else nodes  # noqa: E731
    kind = lambda f: torch.float64 if f == "pr" else torch.int8 if f == "markt" else torch.float32  # noqa: E731
    return {f: _pinned(size(f), kind(f)) for f in names}


def _outputs(case):
    return {"stokes": FLOW, "heat": ("tk", "markk"), "markers": NODES + MOVED,
            "step": FLOW + NODES + MOVED}[case["kind"]]


def prepare(case, seed):
    if case["kind"] == "unet":
        return _prepare_net(case, seed)
    kind = case["kind"]
    mode = _mode(case)
    buf = abi.ModelBuffers(_image(case, seed))
    params = abi.make_params(mode, stokes_rtol=1e-8, stokes_maxcyc=3000, heat_rtol=1e-10, precision=case.get("precision", 1),
                             krylov=case.get("krylov", 0), warm_start=case.get("warm_start", 1), marker_exact=case.get("marker_exact", 0))
    ctx = lib.Context(buf, params, abi.make_file_params(mode.files[0]))
    ctx.prepare()
    n, m = buf.prn.nodenum, buf.prn.marknum
    if kind == "markers":
        flow = dict(zip(("vx", "vy", "vz"), _roll(case)))
        ctx.call("i3g_upload", _part(buf.model, tuple(flow), flow), abi.SYNC_NODES)
        ctx.call("i3g_stokes_stresses")
    state = {"case": case, "ctx": ctx, "mode": mode}
    if kind in ("stokes", "step"):
        # the restart: what a run reads from its file
        names = FLOW if kind == "stokes" else FLOW + abi.NODE_F32[3:] + abi.MARK_F32 + ("markt",)
        state["restart"] = _space(names, n, m)
        state["up"] = _part(buf.model, names, state["restart"])
        ctx.call("i3g_download", state["up"], abi.SYNC_NODES | (abi.SYNC_MARKERS if kind == "step" else 0))
    names = _outputs(case)
    state["out"] = _space(names, n, m)
    state["down"] = _part(buf.model, names, state["out"])
    # the context has its own copy of the image: let go of the large arrays
    buf.f32, buf.prn, buf.markt = {}, None, None
    return state


def run(state):
    if "net" in state:
        out, loss, grads = state["net"].eval_host(state["in5"], state["tg4"] if state["grads"] else None, state["grads"])
        return {"out": out, "loss": loss, "grads": grads} if state["grads"] else {"out": out}
    ctx, mode = state["ctx"], state["mode"]
    plan = mode.files[0]
    kind = state["case"]["kind"]
    marks = abi.SYNC_MARKERS if kind in ("heat", "markers", "step") else 0
    if "up" in state:
        ctx.call("i3g_upload", state["up"], abi.SYNC_NODES | (marks and marks | abi.SYNC_ASYNC))
    for n0 in range(plan.cyc0max):
        runtime.time_step(ctx, mode, plan, n0)
    ctx.call("i3g_download", state["down"], abi.SYNC_NODES | marks)
    return _as_file(state["out"])


def _as_file(out):
    """The fields as the restart file keeps them: pressure in FP32."""
    return dict(out, pr=out["pr"].astype(np.float32)) if "pr" in out else dict(out)


def work(case):
    """What a pass cannot do without: every input read once, every output written once, per time step."""
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "unet":
        # per layer: level, channels in and out, channels of the skip tensor
        flops = byte = 0
        for level, cin, cout, skip in _LAYERS:
            rows = math.prod((v - 1) // 2 ** level + 1 for v in (case["nx"], case["ny"], case["nz"]))
            cin_, cout_ = min(cin, 5) if (level, cin) == (0, 16) and not flops else cin, cout
            flops += rows * 54 * cin_ * cout_
            byte += rows * 2 * (cin + cout + skip) + 54 * cin * cout
        return {"bytes": byte * (3 if case["grads"] else 1), "flops": flops * (3 if case["grads"] else 1)}
    cells = (case["nx"] - 1) * (case["ny"] - 1) * (case["nz"] - 1)
    m = cells * case["mnum"] ** 3
    steps = case.get("steps", 1)
    # nodes: 5 viscosities, density, v, P in; v, P out
    stokes = n * (6 * 4 + 20 + 20)
    # nodes: T, k, rho, cp in, T out; markers: position, type and temperature in, temperature out
    heat = n * 20 + m * 21
    # markers: 25 B read, position, temperature, viscosity, strain written; 13 nodal fields in, 12 out
    moved = m * (25 + 24) + n * (13 * 4 + 12 * 4)
    byte = {"stokes": stokes, "heat": steps * heat, "markers": steps * moved, "step": steps * (stokes + heat + moved)}[case["kind"]]
    # one application of the operator, 4 rows of 17 coefficients per node; RK4: 4 x 3 trilinear sums per marker
    flops = {"stokes": n * 140, "heat": steps * (n * 20 + m * 100), "markers": steps * m * 400,
             "step": steps * (n * 160 + m * 500)}[case["kind"]]
    return {"bytes": byte, "flops": flops}


# ---------------------------------------------------------------------------------------
# the network of the learned warm start
# ---------------------------------------------------------------------------------------
# level, channels in, channels out, channels of the skip tensor
_LAYERS = ((0, 16, 16, 0), (0, 16, 16, 0), (1, 16, 32, 0), (1, 32, 32, 0), (2, 32, 64, 0), (2, 64, 64, 0), (3, 64, 128, 0),
           (3, 128, 128, 0), (2, 128, 64, 64), (2, 64, 64, 0), (1, 64, 32, 32), (1, 32, 32, 0), (0, 32, 16, 16), (0, 16, 16, 0),
           (0, 16, 16, 0))
_SCALES = (21.0, 0.5, 3300.0, 0.0125, 1e-10, 1e6)


def _weights(seed):
    """He-scaled random weights and small biases, flat as the library keeps them: per layer W[27][out][in], b[out]."""
    rng = np.random.default_rng(seed)
    out = []
    for q, (_, cin, cout, _) in enumerate(_LAYERS):
        used = 5 if q == 0 else cin
        w = rng.normal(0, math.sqrt(2.0 / (27 * used)), (27, cout, cin)).astype(np.float32)
        w[:, :, used:] = 0
        out += [w.reshape(-1), rng.normal(0, 0.05, cout).astype(np.float32)]
    return np.concatenate(out)


def _sample(case, seed):
    """log10 viscosity, density and start velocity with warm and stiff blobs, and a smooth correction."""
    rng = np.random.default_rng(seed)
    dims = case["nz"], case["nx"], case["ny"]
    z, x, y = np.meshgrid(*(np.linspace(0, 1, n) for n in dims), indexing="ij")
    a = rng.uniform(2, 5, 12)
    le = 21 + 1.5 * np.sin(a[0] * x + a[1] * y) * np.cos(a[2] * z)
    ro = 3300 + 60 * np.cos(a[3] * y + a[4] * x)
    for _ in range(8):
        c, r = rng.uniform(0.1, 0.9, 3), rng.uniform(0.05, 0.2)
        inside = (z - c[0]) ** 2 + (x - c[1]) ** 2 + (y - c[2]) ** 2 < r * r
        le[inside] += rng.uniform(-1, 1)
        ro[inside] += rng.uniform(-50, 50)
    v = [1e-10 * np.sin(a[5 + k] * x + k * y + z) for k in range(3)]
    d = [1e6 * np.cos(a[8] * x + z)] + [1e-10 * np.cos(a[9 + k] * z + x + k * y) for k in range(3)]
    flat = lambda fields: np.stack([f.reshape(-1) for f in fields]).astype(np.float32)  # noqa: E731
    return flat([le, ro] + v), flat(d)


def _prepare_net(case, seed):
    net = UNet(case["nx"], case["ny"], case["nz"], capacity=1, seed=1)
    net.set_params(_weights(seed))
    net.set_scales(*_SCALES)
    in5, tg4 = _sample(case, seed)
    return {"net": net, "in5": in5, "tg4": tg4, "grads": case["grads"]}


def _exact_net(case, seed):
    """The same network in 64 bits (the library computes with BF16 operands)."""
    import torch.nn.functional as F
    par = torch.from_numpy(_weights(seed)).cuda().double().requires_grad_(case["grads"])
    in5, tg4 = (torch.from_numpy(a).cuda().double() for a in _sample(case, seed))
    dims = case["nz"], case["nx"], case["ny"]
    layers, at = [], 0
    for _, cin, cout, _ in _LAYERS:
        w = par[at:at + 27 * cin * cout].reshape(3, 3, 3, cout, cin).permute(3, 4, 0, 1, 2)
        at += 27 * cin * cout
        layers.append((w, par[at:at + cout]))
        at += cout
    em, ei, rm, ri, vs, ps = _SCALES
    x = torch.zeros(1, 16, *dims, dtype=torch.float64, device="cuda")
    x[0, :5] = torch.stack([(in5[0] - em) * ei, (in5[1] - rm) * ri, *(in5[2:] / vs)]).reshape(5, *dims)
    k1 = torch.tensor([0.25, 0.5, 0.25], dtype=torch.float64, device="cuda")
    k3 = (k1[:, None, None] * k1[None, :, None] * k1[None, None, :])[None, None]

    def conv(q, a, skip=None, relu=True):
        r = F.conv3d(a, layers[q][0], layers[q][1], padding=1)
        r = r if skip is None else r + skip
        return F.relu(r) if relu else r

    def down(a):
        c = a.shape[1]
        return F.conv3d(a, k3.expand(c, 1, 3, 3, 3), stride=2, padding=1, groups=c)

    def up(a):
        return F.interpolate(a, size=[2 * n - 1 for n in a.shape[2:]], mode="trilinear", align_corners=True)
    with torch.enable_grad():
        e0 = conv(1, conv(0, x))
        e1 = conv(3, conv(2, down(e0)))
        e2 = conv(5, conv(4, down(e1)))
        b = conv(7, conv(6, down(e2)))
        g = conv(9, conv(8, up(b), e2))
        g = conv(11, conv(10, up(g), e1))
        g = conv(13, conv(12, up(g), e0))
        y = conv(14, g, relu=False)[0, :4].reshape(4, -1)
        scale = torch.tensor([ps, vs, vs, vs], dtype=torch.float64, device="cuda")[:, None]
        if not case["grads"]:
            return {"out": (y * scale).detach().cpu().numpy()}
        loss = ((y - tg4 / scale) ** 2).mean()
        grad = torch.autograd.grad(loss, par)[0].clone()
    first = grad[:27 * 256].reshape(27, 16, 16)
    first[:, :, 5:] = 0   # the padding channels take no part
    return {"out": (y * scale).detach().cpu().numpy(), "loss": float(loss), "grads": grad.cpu().numpy()}


# ---------------------------------------------------------------------------------------
# markers and heat in 64 bits
# ---------------------------------------------------------------------------------------
class _Exact:
    """The marker and heat steps of a model on uniform grid lines in plain FP64 torch."""

    def __init__(self, case, seed):
        self.case = case
        self.dims = case["nx"], case["ny"], case["nz"]
        self.size, self.h = _size(case)
        pos, types, temp, rocks = _markers(case, seed)
        self.p = [a.double() for a in pos]
        self.t, self.k = types, temp.double()
        self.table = torch.zeros(32, 4, dtype=torch.float64, device="cuda")
        for t, r in rocks.items():
            self.table[t] = torch.tensor([r.nu, r.dh, r.ro, r.kt], dtype=torch.float64)
        self.clamp = (rocks[model.MATRIX].n0, rocks[model.MATRIX].n1)
        self.v = None
        self.f = {}
        y = torch.arange(self.dims[1], device="cuda", dtype=torch.float64) * self.h
        full = (self.dims[2], self.dims[0], self.dims[1])
        self.f["tk"] = (T_TOP + (T_BOTTOM - T_TOP) * y / self.size[1]).expand(full).clone()

    def viscosity(self):
        nu, dh = self.table[self.t.long(), 0], self.table[self.t.long(), 1]
        v = nu * torch.exp(torch.clamp(dh / (RGAS * self.k), max=150.0))
        return v.clamp(max(self.clamp[0], 1e18), min(self.clamp[1], 1e24))

    def stencil(self, p, shift=0.0, lo=0, hi=None):
        """First index and weight of the second one per axis; nodes at (i + shift) * h, index in [lo, hi]."""
        out = []
        for q, a in enumerate(p):
            s = shift[q] if isinstance(shift, tuple) else shift
            u = a / self.h - s
            i = u.floor().clamp(lo, (self.dims[q] - (2 if s == 0 else 3)) if hi is None else hi)
            out.append((i.long(), u - i))
        return out

    def corners(self, st):
        (ix, wx), (iy, wy), (iz, wz) = st
        nx, ny, _ = self.dims
        for c in range(8):
            dz, dx, dy = c >> 2, (c >> 1) & 1, c & 1
            w = (wx if dx else 1 - wx) * (wy if dy else 1 - wy) * (wz if dz else 1 - wz)
            yield ((iz + dz) * nx + ix + dx) * ny + iy + dy, w

    def at(self, f, st):
        f = f.reshape(-1)
        return sum(f[n] * w for n, w in self.corners(st))

    def nodes(self):
        """Marker -> node averages (arithmetic viscosity averages) and the temperature rows."""
        nx, ny, nz = self.dims
        N = nx * ny * nz
        inside = (self.p[0] > 0) & (self.p[1] > 0) & (self.p[2] > 0)
        for q in range(3):
            inside &= self.p[q] < self.size[q]
        t = self.t.long()
        v = self.viscosity() if self.v is None else self.v
        self.v = v
        x, y, z = self.p
        soft = (y < 5e4) & (x > self.size[0] - 1e4) & (z > 1.5e5) & (z < 8.7e5) & (v > 1e19)
        v = torch.where(soft, torch.full_like(v, 1e19), v)
        st = self.stencil(self.p)
        sums = {k: torch.zeros(N, dtype=torch.float64, device="cuda") for k in
                ("w", "ro", "cp", "kt", "tk", "wnu", "nu", "wxx", "nxx", "wxy", "nxy", "wxz", "nxz", "wyz", "nyz")}
        (ix, wx), (iy, wy), (iz, wz) = st
        ro, kt = self.table[t, 2], self.table[t, 3]
        for c, (n, w) in enumerate(self.corners(st)):
            dz, dx, dy = c >> 2, (c >> 1) & 1, c & 1
            w = torch.where(inside, w, torch.zeros_like(w))
            a = wx if dx else 1 - wx
            b = wy if dy else 1 - wy
            d = wz if dz else 1 - wz
            for k, q in (("w", None), ("ro", ro), ("cp", 1000.0 * ro), ("kt", kt), ("tk", self.k), ("wnu", None), ("nu", v)):
                sums[k].index_add_(0, n, w if q is None else w * q)
            tent = lambda s: 0.5 - (s - 0.5).abs()  # noqa: E731
            half = lambda s: (s - 0.5).clamp(min=0)  # noqa: E731
            kinds = []
            if dx and dy and dz:
                kinds.append(("xx", tent(a) * tent(b) * tent(d)))
            if not dz:
                kinds.append(("xy", half(a) * half(b) * tent(d)))
            if not dy:
                kinds.append(("xz", half(a) * tent(b) * half(d)))
            if not dx:
                kinds.append(("yz", tent(a) * half(b) * half(d)))
            for k, g in kinds:
                g = torch.where(inside, 8.0 * g, torch.zeros_like(g))
                sums["w" + k].index_add_(0, n, g)
                sums["n" + k].index_add_(0, n, g * v)
        full = (nz, nx, ny)

        def mean(name, s, w):
            old = self.f.get(name, torch.zeros(full, dtype=torch.float64, device="cuda")).reshape(-1)
            self.f[name] = torch.where(sums[w] > 0.01, s / sums[w].clamp(min=1e-300), old).reshape(full)
        for k in ("xx", "xy", "xz", "yz"):
            mean("n" + k, sums["n" + k], "w" + k)
        mean("nu", sums["nu"], "wnu")
        self.f["nu"] = self.f["nu"].clamp(1e18, 1e24)
        mean("ro", sums["ro"], "w")
        for k in ("kt", "tk"):
            mean(k, sums[k], "w")
        mean("cp", sums["cp"] / self.f["ro"].reshape(-1).clamp(min=1e-300), "w")
        old = self.f["tk"]
        self.f["tk"] = new = old.clone()
        new[:, 0], new[:, -1], new[0], new[-1] = old[:, 1], old[:, -2], old[1], old[-2]
        new[:, :, 0], new[:, :, -1] = T_TOP, T_BOTTOM

    def velocity(self, flow, p):
        p = [a.clamp(0.0, s) for a, s in zip(p, self.size)]
        out = []
        for q, f in enumerate(flow):
            shift = tuple(0.0 if a == q else 0.5 for a in range(3))
            out.append(self.at(f, self.stencil(p, shift)))
        return out

    def move(self, flow, dt):
        self.v = self.viscosity()
        p = self.p
        v1 = self.velocity(flow, p)
        v2 = self.velocity(flow, [a + 0.5 * dt * b for a, b in zip(p, v1)])
        v3 = self.velocity(flow, [a + 0.5 * dt * b for a, b in zip(p, v2)])
        v4 = self.velocity(flow, [a + dt * b for a, b in zip(p, v3)])
        self.p = [a + dt * (b + 2 * c + 2 * d + e) / 6 for a, b, c, d, e in zip(p, v1, v2, v3, v4)]

    @staticmethod
    def with_walls(u):
        """Inner temperatures with the boundary rows: fixed top and bottom, insulating sides."""
        full = torch.empty([n + 2 for n in u.shape], dtype=u.dtype, device=u.device)
        full[1:-1, 1:-1, 1:-1] = u
        full[:, 0], full[:, -1] = full[:, 1], full[:, -2]
        full[0], full[-1] = full[1], full[-2]
        return full

    def heat(self, dt):
        f, h = self.f, self.h
        k, old = f["kt"], f["tk"]
        rocp = (f["ro"] * f["cp"])[1:-1, 1:-1, 1:-1]
        mid = k[1:-1, 1:-1, 1:-1]
        inner = (slice(1, -1),) * 3

        def side(a, axis, by):
            s = list(inner)
            s[axis] = slice(1 + by, a.shape[axis] - 1 + by)
            return a[tuple(s)]

        def apply(u, top, bottom):
            full = self.with_walls(u)
            full[:, :, 0], full[:, :, -1] = top, bottom
            r = rocp / dt * u
            for axis in range(3):
                for by in (-1, 1):
                    r = r - 0.5 * (mid + side(k, axis, by)) / h ** 2 * (side(full, axis, by) - u)
            return r
        u = old[inner].clone()
        r = rocp / dt * u - apply(u, T_TOP, T_BOTTOM)
        d, rr, stop = r.clone(), (r * r).sum(), 1e-28 * ((rocp / dt * u) ** 2).sum()
        for _ in range(1000):
            if rr <= stop:
                break
            ad = apply(d, 0.0, 0.0)
            a = rr / (d * ad).sum()
            u += a * d
            r -= a * ad
            rr, last = (r * r).sum(), rr
            d = r + rr / last * d
        new = self.with_walls(u)
        new[:, :, 0], new[:, :, -1] = T_TOP, T_BOTTOM
        f["tk"] = new
        # markers: nodal change plus the subgrid part, whose mean over each node is taken back
        inside = torch.ones_like(self.k, dtype=torch.bool)
        for p, s in zip(self.p, self.size):
            inside &= (p > 0) & (p < s)
        st = self.stencil(self.p)
        e2, e3 = self.at(new, st), self.at(old, st)
        kt, rc = self.at(k, st), self.at(f["ro"] * f["cp"], st)
        most = torch.stack([new.reshape(-1)[n] for n, _ in self.corners(st)]).amax(0)
        edge = torch.zeros_like(inside)
        for (i, _), n in zip(st, self.dims):
            edge |= (i <= 0) | (i >= n - 2)
        mk = torch.where(edge & (self.k + e2 - e3 > most), most - e2 + e3, self.k)
        sub = (e3 - mk) * (1 - torch.exp((-kt / rc * 6 / h ** 2 * dt).clamp(min=-150.0)))
        N = new.numel()
        a0, a1 = (torch.zeros(N, dtype=torch.float64, device="cuda") for _ in range(2))
        for n, w in self.corners(st):
            w = torch.where(inside, w, torch.zeros_like(w))
            a0.index_add_(0, n, w)
            a1.index_add_(0, n, w * sub)
        back = self.at(a1 / torch.where(a0 == 0, torch.ones_like(a0), a0), st)
        self.k = torch.where(inside, mk + sub + e2 - e3 - back, self.k)


def exact(case, seed):
    """64-bit results of the heat, marker and network cases.  A Stokes solve has no closed form in reach
    here (its matrix needs a sparse direct solver), so the solves and whole segments give none; nor has the
    yielding model, whose viscosity depends on a solve's pressure."""
    if case["kind"] == "unet":
        return _exact_net(case, seed)
    if case["kind"] not in ("heat", "markers") or case["model"] == "plastic":
        return None
    e = _Exact(case, seed)
    e.nodes()
    e.nodes()   # the initial-condition passes average twice
    dt = _mode(case).files[0].maxtmstep_yr * YEAR
    host = lambda a: a.reshape(-1).cpu().numpy()  # noqa: E731
    if case["kind"] == "heat":
        for _ in range(case["steps"]):
            e.heat(dt)
        return {"tk": host(e.f["tk"]), "markk": host(e.k)}
    flow = [torch.from_numpy(a).cuda().double().reshape(case["nz"], case["nx"], case["ny"]) for a in _roll(case)]
    for _ in range(case["steps"]):
        e.move(flow, dt)
        e.nodes()
    out = {f: host(e.f[f]) for f in NODES}
    # strains and formation times stay what they are: no marker yields, none is hydrated
    out.update(markx=host(e.p[0]), marky=host(e.p[1]), markz=host(e.p[2]), markk=host(e.k), markv=host(e.v), marke=None,
               markft=None, markt=None)
    return out
