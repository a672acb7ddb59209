"""The work a user of this framework has it do, as cases that can be timed.

Each case is one pass through the public entry points, over the range of
sizes, storage forms and boundary schemes that the configurations, tests and
the benchmark of this repository use:

* ``flow``: time steps of one flow case - a lid-driven cavity in 2D or 3D, a
  force-driven channel, the three-block L-shaped channel - followed by the
  check-period work of the iteration loop (moments, residual) and the copy of
  the moments to pinned host memory.  ``calls = "loop"`` gives all steps of a
  check period in one call, as ``Solver.iterate`` does; ``calls = "each"``
  makes one call per time step, as the reference's own time loop does through
  the drop-in.
* ``cavities``: a batch of independent cavities of uneven sizes started from
  given fields and run over a few check periods.
* ``predict`` and ``train``: the warm-start network's inference and its
  training steps.
* ``layer``: one convolution of that network by itself: forward, data gradient
  and weight gradient.

``exact`` restates the arithmetic in plain 64-bit torch where that is short
enough: cavities and channels of one block, the batch, and the network.
"""
import ctypes
import itertools
import math

import numpy as np
import torch

from mplb_b200 import abi, config, warmstart
from mplb_b200.batch import Batch, CavitySpec, cavity_set
from mplb_b200.solver import Solver

SQRT3 = math.sqrt(3.0)

#: (side, input channels, output channels, taps) of the network's convolutions
LAYERS = [(128, 32, 32, 9), (128, 32, 32, 9), (64, 32, 64, 9), (64, 64, 64, 9),
          (32, 64, 128, 9), (32, 128, 128, 9), (16, 128, 256, 9), (16, 256, 256, 9),
          (32, 384, 128, 9), (32, 128, 128, 9), (64, 192, 64, 9), (64, 64, 64, 9),
          (128, 96, 32, 9), (128, 32, 32, 9), (128, 32, 16, 1)]


# --------------------------------------------------------------------------
# the cases
def flow(name, family, size, precision, steps, periods=1, wall="EQMDiffuseRefl",
         scheme="Scheme_StreamCollision", calls="loop"):
    nx, ny, nz = size
    case = dict(kind="flow", family=family, nx=nx, ny=ny, nz=nz, precision=precision,
                steps=steps, periods=periods, wall=wall, scheme=scheme, calls=calls)
    return dict(case, name=name) if name else case


def listed():
    swap = "Scheme_StreamCollision_Swap"
    hbb = "HalfwayBounceBack"
    return [
        # the reference's own 2D cavity: its time loop makes one call a step,
        # the smallest calls there are
        flow("cavity2d-128-fp64-each", "cavity2d", (128, 128, 1), "fp64", 200, calls="each"),
        # a small 3D cavity run by the check period: launches and latency
        # count as much as bandwidth
        flow("cavity3d-64-fp64", "cavity3d", (64, 64, 64), "fp64", 300),
        # the benchmark's cavity in its three storage forms, FP16 on an odd side
        flow("cavity3d-256-fp64", "cavity3d", (256, 256, 256), "fp64", 100),
        flow("cavity3d-256-fp32", "cavity3d", (256, 256, 256), "fp32", 100),
        flow("cavity3d-231-fp16", "cavity3d", (231, 231, 231), "fp16", 100),
        # one population array instead of two
        flow("cavity3d-192-fp64-swap", "cavity3d", (192, 192, 192), "fp64", 100, scheme=swap),
        # three joined blocks, periodic in z, perturbed inlet, pressure outlet
        flow("lchannel-384-fp64", "lchannel", (384, 128, 128), "fp64", 60),
        # the precision study's wide 2D channel: periodic, body force, halfway walls
        flow("channel2d-4096-fp32", "channel2d", (4096, 1024, 1), "fp32", 300, wall=hbb),
        # the batch workload, and a small one of ragged sizes in 64 bits
        dict(kind="cavities", name="cavities-4096-fp32", count=4096, precision="fp32",
             sizes="64,96,128,192,256", check=100, periods=2),
        dict(kind="cavities", name="cavities-60-fp64", count=60, precision="fp64",
             sizes="33,64,97,128,200", check=200, periods=2),
        # predictions for a few hundred cavities, and training mini-batches
        dict(kind="predict", name="predict-256", count=256, batch=32),
        dict(kind="train", name="train-32", samples=128, batch=32, steps=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


#: node updates of a drawn flow or batch pass
NODE_STEPS = 1.2e9


def draw(rng):
    kind = rng.choice(["cavity2d", "cavity3d", "cavity3d", "channel2d", "channel3d", "lchannel",
                       "cavities", "cavities", "predict", "train", "layer"])
    if kind == "cavities":
        precision = rng.choice(["fp32", "fp32", "fp64"])
        sizes = sorted(rng.sample(range(24, 257), 3) + rng.sample([64, 96, 128, 192, 256], 2))
        count = _log(rng, 4, 2048 if precision == "fp32" else 512)
        return dict(kind="cavities", count=count, precision=precision,
                    sizes=",".join(map(str, sizes)), check=rng.randrange(20, 101), periods=2)
    if kind == "predict":
        return dict(kind="predict", count=_log(rng, 1, 240), batch=rng.choice([8, 16, 32]))
    if kind == "train":
        return dict(kind="train", samples=rng.randrange(48, 200), batch=_log(rng, 4, 40), steps=3)
    if kind == "layer":
        side = rng.choice([16, 32, 64, 128])
        width = 4096 // side
        return dict(kind="layer", images=_log(rng, 2, 32), side=side,
                    cin=rng.choice([width // 2 * 2, width, width // 2 * 3, 32]),
                    cout=rng.choice([width, width // 2, 16]), taps=rng.choice([9, 9, 9, 1]))
    precision = rng.choice(["fp64", "fp64", "fp32", "fp16"])
    wall = rng.choice(["EQMDiffuseRefl", "EQMDiffuseRefl", "HalfwayBounceBack"])
    scheme, calls = "Scheme_StreamCollision", rng.choice(["loop", "loop", "loop", "each"])
    if kind == "cavity2d":
        n = _log(rng, 24, 2048)
        size = (n, n, 1)
    elif kind == "cavity3d":
        n = _log(rng, 20, 250)
        size = (n, n, n)
        if rng.random() < 0.25:
            scheme, wall = "Scheme_StreamCollision_Swap", "EQMDiffuseRefl"
    elif kind == "channel2d":
        size = (_log(rng, 48, 4096), _log(rng, 32, 1024), 1)
    elif kind == "channel3d":
        size = (_log(rng, 24, 400), _log(rng, 24, 200), _log(rng, 24, 200))
    else:
        side = rng.randrange(24, 129)
        size = (side * rng.randrange(2, 4), side, rng.randrange(24, 129))
        wall = "EQMDiffuseRefl"
    nodes = math.prod(size) * (2 if kind == "lchannel" else 1)
    most = 150 if calls == "each" else 400
    steps = max(10, min(most, int(NODE_STEPS / nodes))) - rng.randrange(0, 5)
    return flow(None, kind, size, precision, steps, wall=wall, scheme=scheme, calls=calls)


# --------------------------------------------------------------------------
# inputs
def flow_config(case):
    size = (case["nx"], case["ny"], case["nz"])
    family, precision = case["family"], case["precision"]
    if family in ("cavity2d", "cavity3d"):
        n = size[0]
        return config.cavity(2 if family == "cavity2d" else 3, n, 0.05,
                             re=400.0 if n >= 96 else 100.0, wall=case["wall"],
                             precision=precision, scheme=case["scheme"])
    if family in ("channel2d", "channel3d"):
        return config.poiseuille(2 if family == "channel2d" else 3, *size,
                                 wall=case["wall"], precision=precision)
    return config.lchannel(*size, precision=precision)


def smooth_fields(shape, count, seed):
    """`count` fields of the given (z, y, x) shape in [-1, 1]: products of
    sines with drawn phases, one to three periods along each axis."""
    gen = torch.Generator().manual_seed(seed)
    out = []
    for _ in range(count):
        f = torch.ones(1, dtype=torch.float64, device="cuda")
        for axis, n in enumerate(shape):
            k, phase = torch.rand(2, generator=gen, dtype=torch.float64).tolist()
            x = torch.arange(n, dtype=torch.float64, device="cuda") / n
            s = torch.sin(2 * math.pi * ((1 + int(3 * k)) * x + phase))
            view = [1] * len(shape)
            view[axis] = n
            f = f * s.reshape(view)
        out.append(f.expand(shape).contiguous())
    return out


def flow_start(case, shape, seed):
    """Initial moments of one block: density within 1 %, velocity components
    within 0.02."""
    r, u, v, w = smooth_fields(shape, 4, seed)
    return [1.0 + 0.01 * r, 0.02 * u, 0.02 * v, 0.02 * w]


def cavity_specs(case, seed):
    """The benchmark's draw of sides, whatever the seed; Reynolds numbers that
    the smallest sizes still resolve and lid speeds from the seed."""
    sizes = [int(s) for s in case["sizes"].split(",")]
    sides = [s.n for s in cavity_set(case["count"], sizes=sizes)]
    drawn = cavity_set(case["count"], seed, re_range=(100.0, 1000.0))
    return [CavitySpec(n, s.re, s.lid) for n, s in zip(sides, drawn)]


def cavity_start(specs, seed):
    """Packed initial moments of a batch (rho, u, v)."""
    gen = torch.Generator().manual_seed(seed)
    draw_ = torch.rand((len(specs), 4), generator=gen, dtype=torch.float64).cuda()
    n = torch.tensor([s.n for s in specs], device="cuda")
    lid = torch.tensor([s.lid for s in specs], dtype=torch.float64, device="cuda")
    which = torch.repeat_interleave(torch.arange(len(specs), device="cuda"), n * n)
    first = torch.cumsum(n * n, 0) - n * n
    k = torch.arange(which.numel(), device="cuda") - first[which]
    side = n[which]
    x = 2 * math.pi * ((k % side).double() / side + draw_[which, 0])
    y = 2 * math.pi * ((k // side).double() / side + draw_[which, 1])
    rho = 1.0 + 0.002 * torch.sin(x) * torch.cos(y)
    u = 0.2 * SQRT3 * lid[which] * torch.cos(x) * torch.sin(y) * draw_[which, 2]
    v = 0.2 * SQRT3 * lid[which] * torch.sin(x) * torch.cos(y) * draw_[which, 3]
    return rho, u, v


def network_params(seed):
    """Flat fp32 parameters: normal weights of variance 2 / fan-in, biases
    within 0.05."""
    gen = torch.Generator().manual_seed(seed)
    parts = []
    for _, ci, co, taps in LAYERS:
        parts.append(torch.randn(co * taps * ci, generator=gen) * math.sqrt(2.0 / (taps * ci)))
        parts.append(0.1 * torch.rand(co, generator=gen) - 0.05)
    return torch.cat(parts)


def network_inputs(case, seed):
    rng = np.random.default_rng(seed)
    count = case["count"] if case["kind"] == "predict" else case["samples"]
    cond = torch.from_numpy(rng.uniform(0, 1, (count, 3)).astype(np.float32)).cuda()
    if case["kind"] == "predict":
        return cond, None, None
    gen = torch.Generator("cuda").manual_seed(seed)
    target = 0.3 * torch.randn((count, abi.NN_GRID, abi.NN_GRID, 3), generator=gen, device="cuda")
    index = [rng.permutation(count)[:case["batch"]].astype(np.int32)
             for _ in range(case["steps"])]
    return cond, target, index


def layer_inputs(case, seed):
    """x, weights, bias, output gradient and the weights of the data gradient
    (taps reversed, channels exchanged)."""
    gen = torch.Generator("cuda").manual_seed(seed)
    n, s, ci, co, t = (case[k] for k in ("images", "side", "cin", "cout", "taps"))

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda")

    x = normal(n, s, s, ci).relu().bfloat16()
    w = (normal(co, t, ci) * math.sqrt(2.0 / (t * ci))).bfloat16()
    bias = 0.1 * normal(co)
    dy = normal(n, s, s, co).bfloat16()
    wd = w.flip(1).permute(2, 1, 0).contiguous()
    return x, w, bias, dy, wd


# --------------------------------------------------------------------------
# prepare and run
def prepare(case, seed):
    return globals()["prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["run_" + state["case"]["kind"]](state)


def prepare_flow(case, seed):
    cfg = flow_config(case)
    solver = Solver(cfg)
    out = {}
    for b in cfg.block_ids:
        nx, ny, nz = cfg.size3(b)
        start = flow_start(case, (nz, ny, nx), seed + b)
        solver.init_macro(b, *[f.cpu().numpy() for f in start[:cfg.space_dim + 1]])
        out[b] = [torch.empty((nz, ny, nx), dtype=torch.float64, pin_memory=True)
                  for _ in range(cfg.space_dim + 1)]
    if case["family"] == "lchannel":
        k, uvw = config.inlet_perturbation(cfg, seed)
        solver.set_boundary_velocity(k, *uvw)
    return {"case": case, "solver": solver, "out": out}


def run_flow(state):
    case, solver = state["case"], state["solver"]
    residual = []
    for _ in range(case["periods"]):
        if case["calls"] == "each":
            for _ in range(case["steps"]):
                solver.stream_collision()
        else:
            solver.stream_collision(case["steps"])
        solver.update_macro_vars()
        residual.append(solver.calc_residual_error(case["steps"])[1])
    for b, fields in state["out"].items():
        ptrs = [f.data_ptr() for f in fields] + [None] * (4 - len(fields))
        solver._check(solver.lib.mplbgpu_download_macro(solver.h, b, *ptrs))
    return {"residual": np.array(residual), "moments": list(state["out"].values())}


def prepare_cavities(case, seed):
    specs = cavity_specs(case, seed)
    return {"case": case, "batch": Batch(specs, case["precision"]),
            "fields": cavity_start(specs, seed)}


def run_cavities(state):
    case, batch = state["case"], state["batch"]
    steps, residual, converged, _ = warmstart.solve(
        batch, case["check"] * case["periods"], case["check"], 1e-10, state["fields"])
    return {"steps": steps, "residual": residual, "converged": converged,
            "moments": warmstart.device_macro(batch)}


def prepare_predict(case, seed):
    net = warmstart.Network(case["batch"])
    net.set_params(network_params(seed).numpy())
    return {"case": case, "net": net, "cond": network_inputs(case, seed)[0]}


def run_predict(state):
    return state["net"].forward(state["cond"])


#: the last learning rate of the training schedule
LEARNING_RATE = 2e-5


def prepare_train(case, seed):
    net = warmstart.Network(case["batch"])
    net.set_params(network_params(seed).numpy())
    cond, target, index = network_inputs(case, seed)
    grads = torch.empty(net.param_count, dtype=torch.float32, pin_memory=True)
    return {"case": case, "net": net, "cond": cond, "target": target, "index": index,
            "grads": grads}


def run_train(state):
    net, index = state["net"], state["index"]
    for i in index[:-1]:
        net.loss_grad(state["cond"], state["target"], i)
        net.adam(LEARNING_RATE)
    loss = net.loss_grad(state["cond"], state["target"], index[-1], want_loss=True)
    net._check(net.lib.mplbnn_get_grads(net.h, state["grads"].data_ptr()))
    net.adam(LEARNING_RATE)
    return {"loss": loss, "grads": state["grads"]}


def prepare_layer(case, seed):
    x, w, bias, dy, wd = layer_inputs(case, seed)
    return {"case": case, "lib": abi.load_library(), "x": x, "w": w, "bias": bias, "dy": dy,
            "wd": wd, "y": torch.empty_like(dy), "dx": torch.empty_like(x),
            "dw": torch.empty(w.shape, device="cuda")}


def run_layer(state):
    lib, taps = state["lib"], state["case"]["taps"]
    stream = torch.cuda.current_stream().cuda_stream

    def view(t):
        return abi.NNView(t.data_ptr(), *t.shape, t.shape[3])

    x, y, dy, dx = (view(state[k]) for k in ("x", "y", "dy", "dx"))
    ptr = {k: state[k].data_ptr() for k in ("w", "wd", "bias", "dw")}
    state["dw"].zero_()
    for rc in (
            lib.mplbnn_conv_forward(ctypes.byref(x), ptr["w"], taps, ptr["bias"], 1,
                                    ctypes.byref(y), 0, None, stream),
            lib.mplbnn_conv_forward(ctypes.byref(dy), ptr["wd"], taps, None, 0,
                                    ctypes.byref(dx), 0, ctypes.byref(x), stream),
            lib.mplbnn_conv_wgrad(ctypes.byref(dy), ctypes.byref(x), taps, ptr["dw"], stream)):
        if rc != abi.OK:
            raise RuntimeError(lib.mplbnn_error().decode())
    return {"y": state["y"], "dx": state["dx"], "dw": state["dw"]}


# --------------------------------------------------------------------------
# what a pass cannot do without
#: floating-point operations of a node update (moments and collision)
NODE_FLOPS = {9: 190.0, 19: 420.0}
WIDTH = {"fp64": 8, "fp32": 4, "fp16": 2}


def work(case):
    """Steps read and write each population of each node once; moments are
    written once a check period and read again with the previous ones for the
    residual.  Layers read their inputs and weights and write their outputs
    once."""
    if case["kind"] == "flow":
        cfg = flow_config(case)
        nodes, q = cfg.nodes(), cfg.q
        steps = case["steps"] * case["periods"]
        moments = 8.0 * (cfg.space_dim + 1) * 4 * case["periods"]
        return {"bytes": nodes * (2.0 * q * WIDTH[case["precision"]] * steps + moments),
                "flops": nodes * NODE_FLOPS[q] * steps}
    if case["kind"] == "cavities":
        nodes = sum(s.n * s.n for s in cavity_specs(case, 1))
        steps = case["check"] * case["periods"]
        return {"bytes": nodes * (18.0 * WIDTH[case["precision"]] * steps + 72 * case["periods"]),
                "flops": nodes * NODE_FLOPS[9] * steps}
    if case["kind"] == "layer":
        n, s, ci, co, t = (case[k] for k in ("images", "side", "cin", "cout", "taps"))
        return {"bytes": n * s * s * (6.0 * ci + 4.0 * co) + 8.0 * t * ci * co,
                "flops": 3 * 2.0 * n * s * s * ci * co * t}
    train = case["kind"] == "train"
    images = case["batch"] * case["steps"] if train else case["count"]
    byte = flop = 0.0
    for side, ci, co, taps in LAYERS:
        flop += 2.0 * side * side * ci * co * taps * (3 if train else 1)
        byte += 2.0 * side * side * (ci + co) * (3 if train else 1)
    return {"bytes": images * byte, "flops": images * flop}


# --------------------------------------------------------------------------
# 64-bit values
def exact(case, seed):
    return globals()["exact_" + case["kind"]](case, seed)


class Lattice:
    """Velocities and weights of D2Q9 and D3Q19 along the axes (x, y[, z])."""

    def __init__(self, dim):
        self.dim = dim
        self.c = [c for c in itertools.product((0, 1, -1), repeat=dim)
                  if sum(map(abs, c)) <= 2]
        weights = {2: (4 / 9, 1 / 9, 1 / 36), 3: (1 / 3, 1 / 18, 1 / 36)}[dim]
        self.w = [weights[sum(map(abs, c))] for c in self.c]
        self.opp = [self.c.index(tuple(-v for v in c)) for c in self.c]

    def feq(self, i, rho, u):
        cu = sum(SQRT3 * c * v for c, v in zip(self.c[i], u))
        return self.w[i] * rho * (1 + cu + 0.5 * (cu * cu - sum(v * v for v in u)))

    def moments(self, f, shift):
        rho = sum(f)
        return rho, [sum(SQRT3 * c[a] * g for c, g in zip(self.c, f) if c[a]) / rho + shift[a]
                     for a in range(self.dim)]

    def pull(self, g, i):
        """g one step along velocity i, periodic; axis x is the last one."""
        axes = [a for a in range(self.dim) if self.c[i][a]]
        if not axes:
            return g.clone()
        return torch.roll(g, [self.c[i][a] for a in axes], [g.dim() - 1 - a for a in axes])


class WallNodes:
    """One face, edge or corner of a block: its nodes, its faces' axes and
    inward signs."""

    def __init__(self, lat, which):
        self.index = (Ellipsis,) + tuple(
            slice(0, 1) if s == 0 else slice(-1, None) if s == 2 else slice(1, -1)
            for s in reversed(which))
        self.faces = [(a, 1 if s == 0 else -1) for a, s in enumerate(which) if s != 1]
        self.inward = [any(sign * c[a] > 0 for a, sign in self.faces) for c in lat.c]
        kinds = []
        for c in lat.c:
            d = [sign * c[a] for a, sign in self.faces]
            if len(d) == 1:
                kinds.append("in" if d[0] < 0 else "out" if d[0] > 0 else "along")
            elif len(d) == 2:
                kinds.append("in" if (d[0] <= 0 and d[1] < 0) or (d[0] < 0 and d[1] == 0)
                             else "out" if (d[0] >= 0 and d[1] > 0) or (d[0] > 0 and d[1] == 0)
                             else "along")
            else:   # the reference labels its corners the other way round
                kinds.append("along" if not any(d) else "out" if max(d) <= 0
                             else "in" if min(d) >= 0 else "along")
        self.kinds = kinds


class OneBlock:
    """A cavity or a channel with halfway walls, stepped in 64 bits."""

    def __init__(self, cfg, moments):
        self.cfg = cfg
        self.lat = lat = Lattice(cfg.space_dim)
        dt, tau = cfg.dt, cfg.tau_ref
        self.omega = dt / (tau + 0.5 * dt)
        accel = cfg.accel[:lat.dim] if cfg.body_force == "BodyForce_1st" else [0.0] * lat.dim
        self.force = [tau * self.omega * w * sum(SQRT3 * v * a for v, a in zip(c, accel))
                      for c, w in zip(lat.c, lat.w)]
        self.shift = [0.5 * dt * a for a in accel]
        self.f = [lat.feq(i, moments[0], moments[1:]) for i in range(len(lat.c))]
        self.old = moments
        walls = [b for b in cfg.boundaries if b.scheme != "MDPeriodic"]
        self.halfway = walls[0].scheme == "HalfwayBounceBack"
        axes = {"Left": 0, "Right": 0, "Bottom": 1, "Top": 1, "Back": 2, "Front": 2}
        self.walls = [(axes[b.surface], 1 if b.surface in ("Left", "Bottom", "Back") else -1,
                       b.given) for b in walls]
        solid = {a for a, _, _ in self.walls}
        self.nodes = [WallNodes(lat, s) for s in itertools.product((0, 1, 2), repeat=lat.dim)
                      if any(v != 1 and a in solid for a, v in enumerate(s))]

    def step(self):
        lat, q = self.lat, len(self.lat.c)
        rho, u = lat.moments(self.f, self.shift)
        cu2 = sum(v * v for v in u)
        g = []
        for i in range(q):
            cu = sum(SQRT3 * c * v for c, v in zip(lat.c[i], u) if c)
            feq = (lat.w[i] * rho) * (1 + cu + 0.5 * (cu * cu - cu2))
            gi = feq + (1 - self.omega) * (self.f[i] - feq)
            g.append(gi + self.force[i] * rho if self.force[i] else gi)
        new = [lat.pull(g[i], i) for i in range(q)]
        for nodes in self.nodes:
            at = nodes.index
            if not self.halfway:   # not streamed: the value that was there
                for i in range(q):
                    if nodes.inward[i]:
                        new[i][at] = self.f[i][at]
            for axis, sign, given in self.walls:
                if (axis, sign) not in nodes.faces:
                    continue
                if self.halfway:
                    for i in range(q):
                        if sign * lat.c[i][axis] > 0:
                            cu = sum(SQRT3 * c * v for c, v in zip(lat.c[i], given))
                            new[i][at] = g[lat.opp[i]][at] + 2 * lat.w[i] * cu
                else:
                    self.diffuse(new, nodes, given)
        self.f = new

    def diffuse(self, f, nodes, given):
        lat, at = self.lat, nodes.index
        by = {k: [i for i in range(len(lat.c)) if nodes.kinds[i] == k]
              for k in ("in", "out", "along")}
        cu = {i: sum(SQRT3 * c * v for c, v in zip(lat.c[i], given)) for i in by["out"]}
        along = {i: lat.feq(i, 1.0, given) for i in by["along"]}
        denom = 1 - sum(2 * lat.w[i] * cu[i] for i in by["out"]) - sum(along.values())
        rho = 2 * sum(f[i][at] for i in by["in"]) / denom
        for i in by["along"]:
            f[i][at] = along[i] * rho
        for i in by["out"]:
            f[i][at] = f[lat.opp[i]][at] + 2 * rho * lat.w[i] * cu[i]

    def moments_and_residual(self):
        rho, u = self.lat.moments(self.f, self.shift)
        now = [rho] + u
        res = [float(((a - b) ** 2).sum() / (a ** 2).sum()) for a, b in zip(now, self.old)]
        self.old = now
        return now, res


def exact_flow(case, seed):
    # joined blocks and the one-array scheme have no short restatement, nor
    # have diffuse walls that meet periodic faces; beyond this many node
    # updates it takes too long
    steps = case["steps"] * case["periods"]
    nodes = case["nx"] * case["ny"] * case["nz"]
    if (case["family"] == "lchannel" or case["scheme"] != "Scheme_StreamCollision"
            or (case["family"].startswith("channel") and case["wall"] != "HalfwayBounceBack")
            or nodes * steps > 2e9):
        return None
    cfg = flow_config(case)
    nx, ny, nz = cfg.size3(0)
    start = flow_start(case, (nz, ny, nx), seed)[:cfg.space_dim + 1]
    if cfg.space_dim == 2:
        start = [f[0] for f in start]
    block = OneBlock(cfg, start)
    residual = []
    for _ in range(case["periods"]):
        for _ in range(case["steps"]):
            block.step()
        now, res = block.moments_and_residual()
        residual.append(res)
    return {"residual": np.array(residual), "moments": [[m.reshape(nz, ny, nx) for m in now]]}


def exact_cavities(case, seed):
    specs = cavity_specs(case, seed)
    steps = case["check"] * case["periods"]
    if sum(s.n * s.n for s in specs) * steps > 2.5e10:
        return None
    lat = Lattice(2)
    fields = cavity_start(specs, seed)
    first = np.cumsum([0] + [s.n * s.n for s in specs])
    out = [torch.empty_like(f) for f in fields]
    residual = np.zeros(len(specs))
    for n in sorted({s.n for s in specs}):
        which = [k for k, s in enumerate(specs) if s.n == n]
        at = torch.cat([torch.arange(first[k], first[k + 1]) for k in which]).cuda()
        now = [f[at].reshape(len(which), n, n) for f in fields]
        dt = 1.0 / ((n - 1) * SQRT3)

        def each(values):
            return torch.tensor(values, dtype=torch.float64, device="cuda")[:, None, None]

        omega = each([dt / (specs[k].tau_ref + 0.5 * dt) for k in which])
        lid = each([SQRT3 * specs[k].lid for k in which])
        f = [lat.feq(i, now[0], now[1:]) for i in range(9)]
        for _ in range(case["periods"]):
            old = now
            for _ in range(case["check"]):
                f = cavity_step(lat, f, omega, lid)
            rho, u = lat.moments(f, (0.0, 0.0))
            now = [rho] + u
            res = torch.stack([((a - b) ** 2).sum((1, 2)) / (a ** 2).sum((1, 2))
                               for a, b in zip(now, old)]).amax(0) / (case["check"] * dt)
        residual[which] = res.cpu().numpy()
        for o, m in zip(out, now):
            o[at] = m.reshape(-1)
    return {"steps": None, "residual": residual, "converged": None, "moments": out}


def cavity_step(lat, f, omega, lid):
    rho, u = lat.moments(f, (0.0, 0.0))
    g = []
    for i in range(9):
        feq = lat.feq(i, rho, u)
        g.append(feq + (1 - omega) * (f[i] - feq))
    new = [lat.pull(g[i], i) for i in range(9)]
    for axis, side in ((0, 0), (0, 1), (1, 0), (1, 1)):   # the top wall last
        at = [slice(None)] * 3
        at[2 - axis] = slice(-1, None) if side else slice(0, 1)
        at = tuple(at)
        for i, c in enumerate(lat.c):
            if c[axis] == (-1 if side else 1):
                push = 2 * lat.w[i] * SQRT3 * c[0] * lid if (axis, side) == (1, 1) else 0.0
                new[i][at] = g[lat.opp[i]][at] + push
    return new


def split_params(flat):
    """The network's weights as (cout, cin, k, k) and biases."""
    out, o = [], 0
    for _, ci, co, taps in LAYERS:
        k = 3 if taps == 9 else 1
        w = flat[o:o + co * taps * ci].reshape(co, k, k, ci).permute(0, 3, 1, 2)
        o += co * taps * ci
        out.append((w, flat[o:o + co]))
        o += co
    return out


def network64(flat, cond):
    """The network's prediction (count, 128, 128, 3) for flat parameters."""
    act = torch.nn.functional
    layers = iter(split_params(flat))

    def conv(x, relu=True):
        w, b = next(layers)
        y = act.conv2d(x, w, b, padding=w.shape[2] // 2)
        return y.relu() if relu else y

    n, side = cond.shape[0], abi.NN_GRID
    mid = (torch.arange(side, dtype=torch.float64, device=cond.device) + 0.5) / side
    planes = [c[:, None, None].expand(n, side, side) for c in cond.double().unbind(1)]
    planes += [mid[None, None, :].expand(n, side, side), mid[None, :, None].expand(n, side, side)]
    x = torch.stack(planes, 1)
    x = torch.cat([x, x.new_zeros((n, 27, side, side))], 1)
    skips = []
    for _ in range(3):
        x = conv(conv(x))
        skips.append(x)
        x = act.avg_pool2d(x, 2)
    x = conv(conv(x))
    for skip in reversed(skips):
        x = conv(conv(torch.cat([act.interpolate(x, scale_factor=2), skip], 1)))
    return conv(x, relu=False)[:, :3].permute(0, 2, 3, 1)


def exact_predict(case, seed):
    cond = network_inputs(case, seed)[0]
    p = network_params(seed).cuda().double()
    with torch.no_grad():
        return torch.cat([network64(p, c) for c in cond.split(16)])


def exact_train(case, seed):
    cond, target, index = network_inputs(case, seed)
    p = network_params(seed).cuda().double()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    for step, which in enumerate(index, 1):
        at = torch.from_numpy(which).long().cuda()
        loss, grad = 0.0, torch.zeros_like(p)
        for part in at.split(8):
            q = p.detach().requires_grad_()
            one = ((network64(q, cond[part]) - target[part].double()) ** 2).sum()
            one = one / (len(at) * target[0].numel())
            grad += torch.autograd.grad(one, q)[0]
            loss += float(one.detach())
        m = 0.9 * m + 0.1 * grad
        v = 0.999 * v + 0.001 * grad * grad
        rate = LEARNING_RATE * math.sqrt(1 - 0.999 ** step) / (1 - 0.9 ** step)
        p = p - rate * m / (v.sqrt() + 1e-8)
    return {"loss": loss, "grads": grad}


def exact_layer(case, seed):
    x, w, bias, dy, _ = layer_inputs(case, seed)
    k = 3 if case["taps"] == 9 else 1
    x64 = x.double().permute(0, 3, 1, 2).requires_grad_()
    w64 = w.double().reshape(case["cout"], k, k, case["cin"]).permute(0, 3, 1, 2).requires_grad_()
    z = torch.nn.functional.conv2d(x64, w64, padding=k // 2)
    dx, dw = torch.autograd.grad(z, (x64, w64), dy.double().permute(0, 3, 1, 2))
    y = (z.detach() + bias.double()[:, None, None]).relu()
    return {"y": y.permute(0, 2, 3, 1), "dx": dx.permute(0, 2, 3, 1) * (x > 0),
            "dw": dw.permute(0, 2, 3, 1).reshape(case["cout"], case["taps"], case["cin"])}
