"""What a program does with this engine, as cases that can be timed.

Every pass goes through the public Python view of the C ABI (dba_b200.Simulation,
dba_b200.Batch).  A pass advances a simulation by `steps` time steps -- the stretch
between two outputs of a run -- and reads its state fields back, and differs in how the
stretch begins:

  fields    from initial host fields (dba_init / dba_init_f32, page-locked for FP32)
  snapshot  from a saved state in page-locked memory (dba_load_state)
  resident  from where the last pass ended (the run continues on the GPU)

Model B and KH runs stay fully active, so a continued run costs the same per step;
a dendrite grows, so its passes restart.
"""
import math

import numpy as np
import torch

import dba_b200

MODEL_FIELDS = {"dendrite": ["p", "T"], "modelb": ["x", "y", "z"], "kh": ["Mass", "Momx", "Momy", "Energy"]}


def _case(name, model, size, block, precision, steps, start, mode="dba", conserved=False, **more):
    nx, ny, nz = size
    c = dict(name=name, model=model, nx=nx, ny=ny, nz=nz, block=block, precision=precision, steps=steps, start=start,
             mode=mode, conserved=conserved)
    c.update(more)
    return c


def listed():
    return [
        # the 512^2 FP64 dendrite with zero-flux walls: a small grid, latency per step counts
        _case("dendrite2d_512_f64", "dendrite", (512, 512, 1), 8, "f64", 1000, "fields", bc=1, radius=60, corner=False),
        # the reference's own 3-D dendrite input: 256^3, FP64, 4^3 blocks, periodic, an output every 1000 steps
        _case("dendrite3d_256_f64_b4", "dendrite", (256, 256, 256), 4, "f64", 1000, "snapshot", bc=0, radius=50,
              corner=False),
        # the large FP32 dendrite: one octant of a crystal growing from a corner of a 512^3 box
        _case("dendrite3d_512_f32", "dendrite", (512, 512, 512), 8, "f32", 800, "fields", bc=1, radius=160, corner=True),
        # a ragged FP32 box advanced in regular mode (every block), as a check run beside DBA does
        _case("dendrite3d_ragged_f32_regular", "dendrite", (200, 136, 104), 8, "f32", 200, "fields", mode="regular",
              bc=1, radius=30, corner=False),
        # conserved Model B, 2048^2 FP32 in 16x16 blocks: the headline workload of bench.py
        _case("modelb2d_2048_f32_conserved", "modelb", (2048, 2048, 1), 16, "f32", 200, "fields", conserved=True,
              share=1.0, eps=1e-3),
        # a ragged FP32 Model B grid of which a part is active
        _case("modelb2d_ragged_f32", "modelb", (1000, 760, 1), 8, "f32", 300, "fields", share=0.4, eps=1e-3),
        # the reference's own Model B input: 256^3, FP64, 4^3 blocks, threshold 1e-6
        _case("modelb3d_256_f64_b4", "modelb", (256, 256, 256), 4, "f64", 10, "resident", share=1.0, eps=1e-6),
        # 3-D Model B in FP32 and 8^3 blocks, every block advanced (regular mode)
        _case("modelb3d_192_f32_regular", "modelb", (192, 192, 192), 8, "f32", 40, "fields", mode="regular", share=1.0,
              eps=1e-6),
        # FP64 conserved Model B in two dimensions: the parity precision with its global mean correction
        _case("modelb2d_768_f64_conserved", "modelb", (768, 768, 1), 16, "f64", 60, "resident", conserved=True,
              share=1.0, eps=1e-6),
        # FP32 KH flow with the CFL time step, developed everywhere
        _case("kh_2048_f32_cfl", "kh", (2048, 2048, 1), 16, "f32", 100, "resident", cfl=True, eps=1.0),
        # the reference's own KH input: 512^2, FP64, 8x8 blocks, fixed step, threshold 0
        _case("kh_512_f64", "kh", (512, 512, 1), 8, "f64", 200, "resident", cfl=False, eps=0.0),
        # a served sweep: dendrites of mixed sizes admitted, advanced together, read and retired
        dict(name="sweep_16_f32", model="sweep", sims=16, edge_min=128, edge_max=512, block=16, threads=128,
             persistent=False, steps=960, precision="f32"),
    ]


def _edge(rng, lo, hi, mult):
    """A multiple of `mult` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(mult, min(hi // mult * mult, int(round(v / mult)) * mult))


def draw(rng):
    kind = rng.choice(["dendrite2d", "dendrite3d", "dendrite3d", "modelb2d", "modelb2d", "modelb3d", "modelb3d", "kh",
                       "kh", "sweep"])
    if kind == "dendrite2d":
        b = rng.choice([4, 8, 16])
        nx, ny = _edge(rng, 96, 1536, b), _edge(rng, 96, 1536, b)
        prec = rng.choice(["f32", "f64"])
        return _case("", "dendrite", (nx, ny, 1), b, prec, rng.randrange(400, 1400), "fields",
                     mode=rng.choice(["dba", "dba", "regular"]), bc=rng.randrange(2),
                     radius=max(10, int(min(nx, ny) * rng.uniform(0.08, 0.3))), corner=False)
    if kind == "dendrite3d":
        prec = rng.choice(["f32", "f64"])
        b = rng.choice([4, 8])
        nx, ny, nz = (_edge(rng, 64, 320 if prec == "f32" else 224, b) for _ in range(3))
        corner = rng.random() < 0.4
        return _case("", "dendrite", (nx, ny, nz), b, prec, rng.randrange(200, 800), "fields" if prec == "f32" else "snapshot",
                     mode=rng.choice(["dba", "dba", "dba", "regular"]), bc=1 if corner else rng.randrange(2),
                     radius=max(10, int(min(nx, ny, nz) * (rng.uniform(0.2, 0.6) if corner else rng.uniform(0.1, 0.3)))),
                     corner=corner)
    if kind == "modelb2d":
        b = rng.choice([4, 8, 16, 32])
        prec = rng.choice(["f32", "f32", "f64"])
        nx, ny = _edge(rng, 128, 2048 if prec == "f32" else 1024, b), _edge(rng, 128, 2048 if prec == "f32" else 1024, b)
        if rng.random() < 0.4 and b != 4:
            nx, ny = (max(32, v // 32 * 32) for v in (nx, ny))
        full = prec == "f64" or rng.random() < 0.5
        return _case("", "modelb", (nx, ny, 1), b, prec, rng.randrange(60, 300) if prec == "f32" else rng.randrange(20, 60),
                     "fields" if prec == "f32" else "resident", mode=rng.choice(["dba", "dba", "regular"]),
                     conserved=rng.random() < 0.5, share=1.0 if full else round(rng.uniform(0.1, 0.7), 3),
                     eps=1e-6 if prec == "f64" else 1e-3)
    if kind == "modelb3d":
        prec = rng.choice(["f32", "f64"])
        b = rng.choice([4, 8])
        nx, ny, nz = (_edge(rng, 48, 256 if prec == "f32" else 192, b) for _ in range(3))
        return _case("", "modelb", (nx, ny, nz), b, prec, rng.randrange(10, 40), "fields" if prec == "f32" else "resident",
                     mode=rng.choice(["dba", "dba", "regular"]), conserved=rng.random() < 0.3, share=1.0, eps=1e-6)
    if kind == "kh":
        prec = rng.choice(["f32", "f64"])
        b = rng.choice([8, 16])
        top = 1536 if prec == "f32" else 768
        return _case("", "kh", (_edge(rng, 128, top, 16), _edge(rng, 128, top, 16), 1), b, prec, rng.randrange(60, 200),
                     "resident", mode=rng.choice(["dba", "dba", "regular"]), conserved=rng.random() < 0.3,
                     cfl=rng.random() < 0.5, eps=rng.choice([0.0, 0.5]))
    return dict(model="sweep", sims=rng.randrange(4, 20), edge_min=96, edge_max=rng.choice([256, 384, 512]),
                block=rng.choice([8, 16]), threads=rng.choice([128, 256]), persistent=rng.random() < 0.5,
                steps=rng.randrange(4, 14) * 96, precision="f32")


# ---- inputs -------------------------------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _params(case):
    """The configuration values of a case beyond its shape (bench.py's workloads, or the reference's inputs)."""
    if case["model"] == "dendrite":
        return dict(dt=5e-5, dx=0.02, dy=0.02, dz=0.02, delta=0.2, tau=0.0003, epsilon=0.01, alpha=0.9, gamma=40.0,
                    Delta=1.15, metric_p=1e-3, metric_T=1e-5, bc=case["bc"], ic_corner=int(case["corner"]))
    if case["model"] == "modelb":
        return dict(dt=0.001, dx=1.0, dy=1.0, dz=1.0, chi_zb=3.0, eps_x=1.0, eps_y=1.0, eps_z=1.0, k_0=1e-4,
                    metric_eps=case["eps"], x0=0.05, y0=0.05, z0=0.45)
    h = 1.0 / case["ny"]
    return dict(dx=h, dy=h, dz=h, dt=0.1 * h, kh_gamma=1.4 if case["cfl"] else 5.0 / 3.0, metric_eps=case["eps"],
                cfl=0.4 if case["cfl"] else 0.0)


def _config(case):
    return dba_b200.config(case["model"], nx=case["nx"], ny=case["ny"], nz=case["nz"], block=case["block"],
                           precision=1 if case["precision"] == "f32" else 0, conserved=int(case["conserved"]),
                           **_params(case))


def _axes(case):
    dev = _device()
    x = torch.arange(case["nx"], device=dev, dtype=torch.float64).view(1, 1, -1)
    y = torch.arange(case["ny"], device=dev, dtype=torch.float64).view(1, -1, 1)
    z = torch.arange(case["nz"], device=dev, dtype=torch.float64).view(-1, 1, 1)
    return x, y, z


def _inputs(case, seed):
    """Initial fields (dendrite p, T; Model B x, y, z; KH rho, p, vx, vy), FP64 tensors of shape (nz, ny, nx)."""
    gen = torch.Generator().manual_seed(seed * 7919 + 17)

    def rnd(*shape):
        return torch.rand(*shape, generator=gen, dtype=torch.float64).tolist()

    dev = _device()
    shape = (case["nz"], case["ny"], case["nx"])
    if case["model"] == "dendrite":
        # a grown crystal: a rough tanh front and the warm layer around it
        x, y, z = _axes(case)
        off = rnd(3)
        if case["corner"]:
            cx = cy = cz = 0.0
        else:
            cx, cy, cz = (case[k] // 2 + 2 * o - 1 for k, o in zip(("nx", "ny", "nz"), off))
        if case["nz"] == 1:
            cz = 0.0
        dx, dy, dz = x - cx, y - cy, z - cz
        r = torch.sqrt(dx * dx + dy * dy + dz * dz).expand(shape)
        th = torch.atan2(dy, dx)
        rough = torch.zeros((), device=dev, dtype=torch.float64)
        for k, (a, ph) in enumerate(zip(rnd(6), rnd(6))):
            rough = rough + 0.012 * (a + 0.3) * torch.cos((k + 3) * th + 2 * math.pi * ph)
        d = r - case["radius"] * (1.0 + rough)
        p = 0.5 * (1.0 - torch.tanh(d / 2.0))
        T = -1.15 + 1.0 * 0.5 * (1.0 - torch.tanh(d / 8.0))
        return [p.contiguous(), T.contiguous()]
    if case["model"] == "modelb":
        g = torch.Generator(device=dev).manual_seed(seed * 7919 + 29)
        fields = [v + 0.02 * (torch.rand(shape, generator=g, device=dev, dtype=torch.float64) - 0.5) for v in (0.05, 0.05, 0.45)]
        if case["share"] < 1.0:      # the rest of the domain is uniform, hence asleep
            x, y, _ = _axes(case)
            (ox, oy) = rnd(2)
            rad = math.sqrt(case["share"] * case["nx"] * case["ny"] / math.pi)
            dx = torch.remainder(x - ox * case["nx"] + case["nx"] / 2, case["nx"]) - case["nx"] / 2
            dy = torch.remainder(y - oy * case["ny"] + case["ny"] / 2, case["ny"]) - case["ny"] / 2
            inside = ((dx * dx + dy * dy) < rad * rad).expand(shape)
            fields = [torch.where(inside, f, torch.full_like(f, v)) for f, v in zip(fields, (0.05, 0.05, 0.45))]
        return [f.contiguous() for f in fields]
    # KH: shear bands with smooth edges and a developed flow of random modes
    x, y, _ = _axes(case)
    x, y = x / case["nx"], y / case["ny"]
    band = (0.5 * (torch.tanh((y - 0.25) / 0.025) - torch.tanh((y - 0.75) / 0.025))).expand(shape)
    vx, vy = (band - 0.5), torch.zeros(shape, device=dev, dtype=torch.float64)
    for a, b, k, l, ph in zip(rnd(10), rnd(10), rnd(10), rnd(10), rnd(10)):
        kx, ky = 1 + int(5 * k), 1 + int(5 * l)
        w = torch.cos(2 * math.pi * (kx * x + ky * y + ph))
        s = (0.15 * (a + 0.5)) / math.hypot(kx, ky)
        vx, vy = vx + s * ky * w, vy - s * kx * w
        band = band + 0.03 * (b - 0.5) * w
    return [(1.0 + band).contiguous(), torch.full(shape, 2.5, device=dev, dtype=torch.float64), vx.contiguous(), vy.contiguous()]


def _host(t, dtype, pin=True):
    h = torch.empty(t.numel(), dtype=dtype, pin_memory=pin and torch.cuda.is_available())
    h.copy_(t.reshape(-1))
    return h


def _sweep_requests(case, seed):
    gen = torch.Generator().manual_seed(seed * 7919 + 41)
    out = []
    for k in range(case["sims"]):
        e, u, a = torch.rand(3, generator=gen, dtype=torch.float64).tolist()
        # the sizes belong to the case, the physics to the seed
        t = ((k * 7) % case["sims"]) / max(1, case["sims"] - 1)
        edge = int(case["edge_min"] * (case["edge_max"] / case["edge_min"]) ** t) // 16 * 16
        out.append(dict(edge=max(32, edge), Delta=0.9 + 0.35 * u, delta=0.08 + 0.16 * a, radius=8.0 + 2.0 * e))
    return out


def _sweep_config(case, q):
    return dba_b200.config("dendrite", nx=q["edge"], ny=q["edge"], nz=1, block=case["block"], precision=1, bc=1, ic=1,
                           ic_radius=q["radius"], ic_width=2.0, dt=5e-5, dx=0.02, dy=0.02, dz=0.02, tau=0.0003,
                           epsilon=0.01, alpha=0.9, gamma=40.0, metric_p=1e-3, metric_T=1e-5, Delta=q["Delta"],
                           delta=q["delta"])


def prepare(case, seed):
    if case["model"] == "sweep":
        reqs = _sweep_requests(case, seed)
        cells = sum(q["edge"] ** 2 for q in reqs)
        b = case["block"]
        batch = dba_b200.Batch(precision=1, block=b, max_slots=case["sims"], block_capacity=cells // (b * b),
                               cell_capacity=cells, threads=case["threads"])
        batch.set_option(dba_b200.BATCH_PERSISTENT, int(case["persistent"]))
        return dict(case=case, batch=batch, configs=[_sweep_config(case, q) for q in reqs])
    f32 = case["precision"] == "f32"
    ic = _inputs(case, seed)
    sim = dba_b200.Simulation(_config(case))
    state = dict(case=case, sim=sim, fields=MODEL_FIELDS[case["model"]], mode=1 if case["mode"] == "dba" else 0)
    n = case["nx"] * case["ny"] * case["nz"]
    dtype = torch.float32 if f32 else torch.float64
    state["out"] = [torch.empty(n, dtype=dtype, pin_memory=True).numpy() for _ in state["fields"]]
    if case["start"] == "fields" and f32:
        state["ic"] = _host(torch.cat([t.reshape(-1) for t in ic]), torch.float32).numpy()
    elif case["start"] == "fields":
        state["ic"] = [t.reshape(-1).cpu().numpy() for t in ic]
    else:
        sim.init([t.reshape(-1).cpu().numpy() for t in ic])
        if case["start"] == "snapshot":
            state["blob"] = torch.empty(sim.state_size(), dtype=torch.uint8, pin_memory=True)
            sim.save_state(state["blob"])
            sim.sync()
    return state


def run(state):
    case = state["case"]
    if case["model"] == "sweep":
        batch = state["batch"]
        slots = [batch.add(c) for c in state["configs"]]
        batch.step(case["steps"])
        tips, steps = batch.tips()
        fields = [np.float32(batch.field(s, q)) for s in slots for q in ("p", "T")]
        for s in slots:
            batch.remove(s)
        return {"tips": np.float32(tips[slots]), "steps": steps[slots], "fields": fields}
    sim = state["sim"]
    f32 = case["precision"] == "f32"
    if case["start"] == "fields":
        sim.init_f32(state["ic"]) if f32 else sim.init(state["ic"])
    elif case["start"] == "snapshot":
        sim.load_state(state["blob"])
    sim.step(case["steps"], state["mode"])
    read = sim.field_f32 if f32 else sim.field
    return {q: read(q, out=o) for q, o in zip(state["fields"], state["out"])}


# ---- what a pass cannot do without ------------------------------------------------------------------

def _active(case):
    """Share of the cells that a step advances, on average."""
    if case["mode"] == "regular":
        return 1.0
    if case["model"] == "modelb":
        return case["share"]
    if case["model"] == "kh":
        return 1.0
    r, w = case["radius"], 25 + case["block"]         # the front and its warm layer
    if case["nz"] == 1:
        band = 2 * math.pi * r * 2 * w
    else:
        band = 4 * math.pi * (r * r + w * w / 3) * 2 * w
    if case["corner"]:
        band /= 4 if case["nz"] == 1 else 8
    return min(1.0, band / (case["nx"] * case["ny"] * case["nz"]))


def work(case):
    if case["model"] == "sweep":
        cells = sum(min(q["edge"] ** 2, 2 * math.pi * 12 * 50) for q in _sweep_requests(case, 0))
        return {"bytes": cells * case["steps"] * 16.0, "flops": cells * case["steps"] * 60.0}
    n = case["nx"] * case["ny"] * case["nz"]
    size = 4 if case["precision"] == "f32" else 8
    nf = len(MODEL_FIELDS[case["model"]])
    updates = n * _active(case) * case["steps"]
    per = {"dendrite": 60 if case["nz"] == 1 else 75, "modelb": 180 if case["nz"] == 1 else 330, "kh": 300}[case["model"]]
    edge = nf * n * size                                  # the fields handed over and back
    return {"bytes": 2.0 * nf * size * updates + edge * (1 if case["start"] == "resident" else 2), "flops": per * updates}


# ---- the same in 64 bits, in plain torch ---------------------------------------------------------------

class _Grid:
    def __init__(self, nx, ny, nz, block, bc):
        self.bc, self.flat = bc, nz == 1
        self.block = (1 if nz == 1 else block, block, block)
        self.nb = (nz // self.block[0], ny // block, nx // block)

    def at(self, f, axis, by):
        """Every cell's neighbour `by` cells up the axis."""
        if f.shape[axis] == 1:
            return f
        g = torch.roll(f, -by, axis)
        if self.bc:                                       # zero flux: the edge cell is its own neighbour
            n = f.shape[axis]
            k = n - 1 if by > 0 else 0
            g.narrow(axis, k, 1).copy_(f.narrow(axis, k, 1))
        return g

    def cells(self, blocks):
        b = self.block
        return blocks.repeat_interleave(b[0], 0).repeat_interleave(b[1], 1).repeat_interleave(b[2], 2)

    def any(self, mask):
        b, n = self.block, self.nb
        return mask.view(n[0], b[0], n[1], b[1], n[2], b[2]).any(5).any(3).any(1)

    def wake(self, hit, diagonal=False):
        out = hit.clone()
        for axis in (0, 1, 2):
            for by in (-1, 1):
                g = torch.roll(hit, by, axis)
                if self.bc:
                    g.narrow(axis, 0 if by > 0 else hit.shape[axis] - 1, 1).zero_()
                out |= g
        if diagonal:
            for a in (-1, 1):
                for b in (-1, 1):
                    out |= torch.roll(hit, (a, b), (1, 2))
        return out


def _exact_dendrite(g, p, T, q, steps, dba):
    Pi = 3.14159
    f0, f1 = 1.0 / (2 * q["dx"]), 1.0 / q["dx"] ** 2
    pa = torch.ones(g.nb, dtype=torch.bool, device=p.device)
    Ta = pa.clone()
    axes = (2, 1) if g.flat else (2, 1, 0)
    for _ in range(steps):
        s2, s4, lap, lapT = 0.0, 0.0, -2.0 * len(axes) * p, -2.0 * len(axes) * T
        for a in axes:
            up, dn = g.at(p, a, 1), g.at(p, a, -1)
            lap = lap + up + dn
            d2 = ((up - dn) * f0) ** 2
            s2, s4 = s2 + d2, s4 + d2 * d2
            lapT = lapT + g.at(T, a, 1) + g.at(T, a, -1)
        sigma = torch.where(s2 <= 1e-6, torch.ones_like(p), 1.0 - q["delta"] * (1.0 - s4 / (s2 * s2)))
        m = -q["alpha"] / Pi * torch.atan(q["gamma"] * sigma * T)
        pn = p + q["dt"] / q["tau"] * (q["epsilon"] ** 2 * f1 * lap + p * (1 - p) * (p - 0.5 + m))
        Tn = T + q["dt"] * f1 * lapT
        if not dba:
            p, T = pn, Tn + pn - p
            continue
        pc, Tc = g.cells(pa), g.cells(Ta)
        Tn = torch.where(pc, Tn + (pn - p), Tn)
        hp = g.any((pn >= q["metric_p"]) & (pn <= 1 - q["metric_p"]) & pc)
        hT = g.any(((Tn - T).abs() >= q["metric_T"]) & Tc)
        p, T = torch.where(pc, pn, p), torch.where(Tc, Tn, T)
        pa, Ta = g.wake(hp), g.wake(hT)
    return p, T


def _lap27(g, f, dx):
    if g.flat:
        r = f + 0.0
        h = g.at(f, 2, 1) + g.at(f, 2, -1)
        faces = h + g.at(f, 1, 1) + g.at(f, 1, -1)
        diag = g.at(h, 1, 1) + g.at(h, 1, -1)
        return (-10.0 / 3.0 * r + 2.0 / 3.0 * faces + diag / 6.0) / dx ** 2
    sx = g.at(f, 2, 1) + g.at(f, 2, -1)
    sy = g.at(f, 1, 1) + g.at(f, 1, -1)
    sxy = g.at(sx, 1, 1) + g.at(sx, 1, -1)
    pl1, pl2 = sx + sy, sxy                                # a plane's 4 faces, its 4 diagonals
    up = lambda v: g.at(v, 0, 1) + g.at(v, 0, -1)          # noqa: E731
    return (-64.0 / 15.0 * f + 7.0 / 15.0 * (pl1 + up(f)) + 0.1 * (pl2 + up(pl1)) + up(pl2) / 30.0) / dx ** 2


def _exact_modelb(g, x, y, z, q, steps, dba, conserved):
    chi = q["chi_zb"]
    act = torch.ones(g.nb, dtype=torch.bool, device=x.device)
    mx = my = mz = None
    logK = math.log(100.0)
    for _ in range(steps):
        b = 1.0 - x - y - z
        lz = _lap27(g, z, q["dx"])
        lb = torch.log(b)
        ux = torch.log(x) - lb - chi * z - q["eps_x"] * _lap27(g, x, q["dx"])
        uy = torch.log(y) - lb - chi * z - q["eps_y"] * _lap27(g, y, q["dx"])
        uz = -0.5 + chi * b - chi * z + torch.log(z) / 2 - lb - q["eps_z"] * lz - logK / 2
        c = g.cells(act) if dba else None
        mx, my, mz = (n if m is None or not dba else torch.where(c, n, m) for n, m in ((ux, mx), (uy, my), (uz, mz)))
        r = q["k_0"] * (torch.exp(mx + my) - torch.exp(2 * mz))
        dt = q["dt"]
        ch = [dt * (_lap27(g, mx, q["dx"]) - r), dt * (_lap27(g, my, q["dx"]) - r), 2 * dt * (_lap27(g, mz, q["dx"]) + r)]
        if dba:
            ch = [torch.where(c, v, torch.zeros_like(v)) for v in ch]
            act = g.wake(g.any((lz.abs() > q["metric_eps"]) & c))
        x, y, z = x + ch[0], y + ch[1], z + ch[2]
        if dba and conserved:
            x, y, z = (f - v.mean() for f, v in zip((x, y, z), ch))
    return x, y, z


def _exact_kh(g, ic, q, steps, dba, conserved):
    h, gam = q["dx"], q["kh_gamma"]
    vol = h * h
    rho, p, u, v = ic
    U = [rho * vol, rho * u * vol, rho * v * vol, (p / (gam - 1) + 0.5 * rho * (u * u + v * v)) * vol]
    act = torch.ones(g.nb, dtype=torch.bool, device=rho.device)
    speed = (torch.sqrt(gam * p / rho) + torch.sqrt(u * u + v * v)).max()
    keep = {}

    def fresh(name, values, c):
        old = keep.get(name)
        keep[name] = values if old is None or c is None else [torch.where(c, n, o) for n, o in zip(values, old)]
        return keep[name]

    def flux(rL, rR, pL, pR, nL, nR, tL, tR):
        eL, eR = (pp / (gam - 1) + 0.5 * r * (a * a + b * b) for pp, r, a, b in ((pL, rL, nL, tL), (pR, rR, nR, tR)))
        r, mn, mt, e = 0.5 * (rL + rR), 0.5 * (rL * nL + rR * nR), 0.5 * (rL * tL + rR * tR), 0.5 * (eL + eR)
        ps = (gam - 1) * (e - 0.5 * (mn * mn + mt * mt) / r)
        C = 0.5 * torch.maximum(torch.sqrt(gam * pL / rL) + nL.abs(), torch.sqrt(gam * pR / rR) + nR.abs())
        return (mn - C * (rL - rR), (e + ps) * mn / r - C * (eL - eR), mn * mn / r + ps - C * (rL * nL - rR * nR),
                mn * mt / r - C * (rL * tL - rR * tR))

    for _ in range(steps):
        dt = q["cfl"] * h / speed if q["cfl"] > 0 else q["dt"]
        c = g.cells(act) if dba else None
        r = U[0] / vol
        a, b = U[1] / U[0], U[2] / U[0]
        W = fresh("W", [r, (U[3] / vol - 0.5 * r * (a * a + b * b)) * (gam - 1), a, b], c)
        gx = [(g.at(w, 2, 1) - g.at(w, 2, -1)) * 0.5 / h for w in W]
        gy = [(g.at(w, 1, 1) - g.at(w, 1, -1)) * 0.5 / h for w in W]
        r, p, a, b = W
        div = gx[2] + gy[3]
        prime = [r - 0.5 * dt * (a * gx[0] + b * gy[0] + r * div), p - 0.5 * dt * (gam * p * div + a * gx[1] + b * gy[1]),
                 a - 0.5 * dt * (a * gx[2] + b * gy[2] + gx[1] / r), b - 0.5 * dt * (a * gx[3] + b * gy[3] + gy[1] / r)]
        metric = sum(t.abs() for t in gx + gy)
        gx, gy, P = fresh("gx", gx, c), fresh("gy", gy, c), fresh("P", prime, c)
        xm = [g.at(w, 2, 1) - 0.5 * h * g.at(s, 2, 1) for w, s in zip(P, gx)]
        xp = [w + 0.5 * h * s for w, s in zip(P, gx)]
        ym = [g.at(w, 1, 1) - 0.5 * h * g.at(s, 1, 1) for w, s in zip(P, gy)]
        yp = [w + 0.5 * h * s for w, s in zip(P, gy)]
        X = fresh("X", list(flux(xm[0], xp[0], xm[1], xp[1], xm[2], xp[2], xm[3], xp[3])), c)
        Y = fresh("Y", list(flux(ym[0], yp[0], ym[1], yp[1], ym[3], yp[3], ym[2], yp[2])), c)
        fx, fy = [X[0], X[2], X[3], X[1]], [Y[0], Y[3], Y[2], Y[1]]       # Mass, Momx, Momy, Energy
        ch = [dt * h * (g.at(s, 2, -1) - s + g.at(t, 1, -1) - t) for s, t in zip(fx, fy)]
        if dba:
            ch = [torch.where(c, s, torch.zeros_like(s)) for s in ch]
            act = g.wake(g.any((metric > q["metric_eps"]) & c), diagonal=True)
        U = [s + t for s, t in zip(U, ch)]
        if dba and conserved:
            U = [s - t.mean() for s, t in zip(U, ch)]
        r, a, b = U[0] / vol, U[1] / U[0], U[2] / U[0]
        p = (U[3] / vol - 0.5 * r * (a * a + b * b)) * (gam - 1)
        speed = (torch.sqrt(gam * p / r) + torch.sqrt(a * a + b * b)).max()
    return U


def _exact_sweep(case, seed):
    tips, steps, fields = [], [], []
    for q in _sweep_requests(case, seed):
        n = q["edge"]
        c = dict(model="dendrite", nx=n, ny=n, nz=1, bc=1, corner=False)
        x, y, _ = _axes(c)
        r = torch.sqrt((x - n // 2) ** 2 + (y - n // 2) ** 2)
        p = 0.5 * (1.0 - torch.tanh((r - q["radius"]) / 2.0))
        T = torch.full_like(p, -q["Delta"])
        par = dict(_params(c), Delta=q["Delta"], delta=q["delta"])
        p, T = _exact_dendrite(_Grid(n, n, 1, case["block"], 1), p, T, par, case["steps"], True)
        col = p[0, :, n // 2].cpu()
        k = next((k for k in range(n // 2, n) if col[k] < 0.5), None)
        tips.append(float("nan") if k is None else float((col[k - 1] - 0.5) / (col[k - 1] - col[k])) + k - 1 - n // 2)
        steps.append(case["steps"])
        fields += [p.cpu().numpy(), T.cpu().numpy()]
    return {"tips": np.array(tips), "steps": np.array(steps), "fields": fields}


def exact(case, seed):
    if case["model"] == "sweep":
        return _exact_sweep(case, seed)
    ic = _inputs(case, seed)
    if case["precision"] == "f32" and case["start"] == "fields":
        ic = [t.float().double() for t in ic]
    q = _params(case)
    g = _Grid(case["nx"], case["ny"], case["nz"], case["block"], q.get("bc", 0))
    dba = case["mode"] == "dba"
    if case["model"] == "dendrite":
        got = _exact_dendrite(g, *ic, q, case["steps"], dba)
    elif case["model"] == "modelb":
        got = _exact_modelb(g, *ic, q, case["steps"], dba, case["conserved"])
    else:
        got = _exact_kh(g, ic, q, case["steps"], dba, case["conserved"])
    return {k: v.cpu().numpy() for k, v in zip(MODEL_FIELDS[case["model"]], got)}
