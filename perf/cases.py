"""Measured cases of the Fire-X step: what a program steps through the public handles (FireXSim,
FireXBatch) and takes back, from an interactive preview grid to the 508^3 configuration.

A case is one pass: advance `steps` fixed steps, then hand the result on. Three ways of taking
it are in use and appear here:

  read    the flow field copied into host memory the program keeps pinned (the call returns when
          it is there);
  stream  the same copy started behind the step, finishing while later work runs;
  device  the three FP16 render volumes, packed at the end of the step and read by a renderer
          on the same GPU, in stream order with the renderer's own work.

States are a burning plume in gently moving air: hot core, fuel at its foot, products above,
ambient air elsewhere, made from the seed alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fire_b200 import FireXBatch, FireXSim, make_options
from fire_b200 import _abi as A

DT = 1.0 / 60.0
PRESSURE = {"auto": A.PRESSURE_AUTO, "warm": A.PRESSURE_WARM_F32, "f16": A.PRESSURE_F16, "cold": A.PRESSURE_COLD_F32}
# grids of the 48-simulation batch and of the served stream
MEMBER_GRIDS = ((64, 96, 64), (96, 144, 96), (128, 192, 128), (160, 240, 160))
EXACT_CELLS = 48 << 20  # past this the float64 step's temporaries outgrow a shared card


def _case(name, x, y, z, sweeps, emitter="spheres", precision="f32", pressure="warm", steps=1, take="device", water=False,
          members=1):
    return dict(name=name, x=x, y=y, z=z, sweeps=sweeps, emitter=emitter, precision=precision, pressure=pressure,
                steps=steps, take=take, water=water, members=members)


def listed():
    return [
        # an editor's preview while a parameter is dragged: one small step, the flow back at once
        _case("preview_32x48x32", 32, 48, 32, 12, emitter="burner", take="read"),
        # the small plain configuration: 64x96x64, 40 + 40 sweeps
        _case("small_64x96x64", 64, 96, 64, 40),
        # several fixed steps per displayed frame, then the frame's flow and divergence norm
        _case("frame_96x144x96", 96, 144, 96, 64, steps=4, take="read"),
        # the reference's default scene with the spray on, on a grid a user typed in
        _case("spray_100x148x92", 100, 148, 92, 64, emitter="burner", pressure="auto", water=True),
        # the HD tier, FP32, every step's flow streamed to the host
        _case("hd_stream_128x192x128", 128, 192, 128, 96, take="stream"),
        # the HD tier with FP16 species storage, rendered on the GPU
        _case("hd_mixed_128x192x128", 128, 192, 128, 96, precision="mixed"),
        # the largest batch member stepped alone: beyond on-chip memory, within L2
        _case("mid_160x240x160", 160, 240, 160, 96),
        # an uneven grid about the largest the server takes, FP16 species
        _case("uneven_188x284x196", 188, 284, 196, 64, precision="mixed"),
        # an offline render on an uneven grid, burner
        _case("offline_300x452x276", 300, 452, 276, 64, emitter="burner"),
        # the large plain configuration: 508^3, 96 + 96 sweeps, FP32 pressure
        _case("large_508x508x508", 508, 508, 508, 96),
        # a heavy grid under the automatic pressure rule: FP16 pressure storage
        _case("heavy_412x616x412", 412, 616, 412, 64, emitter="burner", pressure="auto"),
        # uneven simulations stepped together, as the server does
        _case("batch_of_12", 0, 0, 0, 96, precision="mixed", members=12),
    ]


def _grid(rng, lo, hi):
    """Axes (multiples of 4, at least 16) of a grid of about lo..hi cells, log-uniform."""
    while True:
        cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        fx, fy, fz = (math.exp(rng.uniform(-0.25, 0.25)) for _ in range(3))
        side = (cells / (1.5 * fx * fy * fz)) ** (1.0 / 3.0)
        d = [max(16, 4 * round(side * f / 4)) for f in (fx, 1.5 * fy, fz)]
        if max(d) <= 1024 and d[0] * d[1] * d[2] <= hi:
            return d


def _unnamed(case):
    del case["name"]
    return case


def draw(rng):
    kind = rng.random()
    sweeps = rng.choice((8, 13, 24, 40, 64, 65, 96))
    if kind < 0.15:  # a batch
        return _unnamed(_case("", 0, 0, 0, rng.choice((40, 64, 96)), precision=rng.choice(("mixed", "f32")),
                              members=rng.randint(2, 12)))
    x, y, z = _grid(rng, 24 << 10, 64 << 20)
    cells = x * y * z
    precision = rng.choice(("f32", "f32", "mixed"))
    take = "device" if cells > (8 << 20) else rng.choice(("read", "stream", "device"))
    return _unnamed(_case("", x, y, z, sweeps, emitter=rng.choice(("burner", "spheres")), precision=precision,
                          pressure=rng.choice(("auto", "warm", "warm", "cold", "f16")),
                          steps=rng.choice((1, 1, 1, 4)) if cells < (2 << 20) else 1, take=take,
                          water=cells < (4 << 20) and rng.random() < 0.15))


# ---- inputs ------------------------------------------------------------------------------------

def _member_dims(case):
    if case["members"] == 1:
        return [(case["x"], case["y"], case["z"])]
    return [MEMBER_GRIDS[(3 * i + i // 4) % 4] for i in range(case["members"])]


def _spheres(case, dims):
    if case["emitter"] != "spheres":
        return None
    X, Y, Z = dims
    r = max(2.0, min(X, Z) / 9.0)
    return [dict(center=(0.5 * X, r * 0.9, 0.5 * Z), radius=r, fuel=1.0, temperature=1500.0)]


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _scene(dims, seed, mixed):
    """(flow, species, pressure) of a plume, float32 on the device, shaped (Z, Y, X[, 4])."""
    dev = _device()
    X, Y, Z = dims
    rnd = np.random.default_rng(seed)
    ax = [(torch.arange(n, device=dev, dtype=torch.float32) + 0.5) / n for n in (X, Y, Z)]
    x, y, z = ax[0].view(1, 1, X), ax[1].view(1, Y, 1), ax[2].view(Z, 1, 1)
    cx, cz, sway = 0.5 + rnd.uniform(-0.06, 0.06), 0.5 + rnd.uniform(-0.06, 0.06), rnd.uniform(0.02, 0.06)
    width = 0.07 + 0.09 * y
    dx = x - cx - sway * torch.sin(7.0 * y + float(rnd.uniform(0, 6)))
    dz = z - cz - sway * torch.cos(6.0 * y + float(rnd.uniform(0, 6)))
    g = torch.exp(-(dx * dx + dz * dz) / (2.0 * width * width)) * torch.exp(-1.2 * y)
    g = torch.where(g > 0.03, g, torch.zeros_like(g))
    flow = torch.empty((Z, Y, X, 4), device=dev, dtype=torch.float32)
    for c in range(3):
        k = rnd.uniform(2.0, 11.0, size=(3, 3))
        ph = rnd.uniform(0.0, 6.28, size=(3, 3))
        v = 0.0
        for m in range(3):
            v = v + 0.06 * (torch.sin(float(k[m, 0]) * x + float(ph[m, 0])) * torch.sin(float(k[m, 1]) * y + float(ph[m, 1]))
                            * torch.sin(float(k[m, 2]) * z + float(ph[m, 2])))
        flow[..., c] = v + (0.6 * g if c == 1 else 0.0)
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    flow[..., :3] += 0.04 * (torch.rand((Z, Y, X, 3), device=dev, generator=gen) - 0.5)
    flow[..., 3] = 300.0 + 1650.0 * g
    species = torch.empty((Z, Y, X, 4), device=dev, dtype=torch.float32)
    species[..., 0] = 0.9 * g * g
    species[..., 1] = 1.0 - 0.7 * g
    species[..., 2] = 0.5 * g
    species[..., 3] = 0.25 * g
    if mixed:
        species = species.half().float()
    pressure = 1e-4 * (flow[..., 0] + flow[..., 1])
    return flow, species, pressure


class _DeviceArray:
    """A device buffer of the library as torch sees it (the array interface torch reads)."""

    def __init__(self, address, shape):
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f2", data=(address, False), version=3)


def _make_sim(case, dims, seed):
    mixed = case["precision"] == "mixed"
    sim = FireXSim(dims, make_options(
        precision=A.PRECISION_MIXED if mixed else A.PRECISION_F32, pressure_mode=PRESSURE[case["pressure"]],
        pressure_iterations=case["sweeps"], correction_iterations=case["sweeps"], spheres=_spheres(case, dims),
        seed=seed, emission_jitter=0.1))
    if case["water"]:
        sim.set_parameter("waterEnabled", True)
        sim.set_parameter("waterFlow", 1.0)
    flow, species, pressure = _scene(dims, seed, mixed)
    sim.write("flow", flow.cpu().numpy())
    sim.write("species", species.cpu().numpy())
    sim.write("pressure", pressure.cpu().numpy())
    return sim


def prepare(case, seed):
    sims = [_make_sim(case, d, seed + 101 * i) for i, d in enumerate(_member_dims(case))]
    state = dict(case=case, sims=sims, stepper=sims[0])
    if case["members"] > 1:
        state["stepper"] = FireXBatch()
        for s in sims:
            state["stepper"].add(s)
    if case["take"] == "device":
        state["volumes"] = []
        for s in sims:
            s.set_render_packing(True)
            X, Y, Z = s.dims
            volumes = [torch.as_tensor(_DeviceArray(p, (Z, Y, X, 4)), device="cuda") for p in s.render_volumes()]
            for v in volumes:
                v.simulation = s  # the buffers live as long as their simulation
            state["volumes"].append(volumes)
        state["stream"] = torch.cuda.ExternalStream(state["stepper"].stream)
    else:
        X, Y, Z = sims[0].dims
        state["flow"] = torch.empty((Z, Y, X, 4), dtype=torch.float32, pin_memory=True).numpy()
    return state


def run(state):
    case, stepper = state["case"], state["stepper"]
    if case["take"] == "device":
        renderer = torch.cuda.current_stream()
        state["stream"].wait_stream(renderer)  # the renderer has finished with the last frame's volumes
        stepper.step(case["steps"], DT)
        renderer.wait_stream(state["stream"])
        return state["volumes"]
    stepper.step(case["steps"], DT)
    if case["take"] == "stream":
        stepper.read_async("flow", state["flow"])
        return {"flow": state["flow"]}
    stepper.read_into("flow", state["flow"])
    if case["steps"] > 1:
        l2, largest, _ = stepper.divergence_norm()
        return {"flow": state["flow"], "norm": l2, "largest": largest}
    return {"flow": state["flow"]}


def work(case):
    """Fields in and out once per step and per Jacobi sweep the arithmetic of one update: the
    sweeps need not touch memory, the step reads flow, species, pressure and liquid and writes
    flow, species, reaction, divergence, pressure and correction."""
    cells = sum(x * y * z for x, y, z in _member_dims(case))
    species = 8 if case["precision"] == "mixed" else 16
    half = case["pressure"] == "f16" or (case["pressure"] == "auto" and cells >= (64 << 20))
    p = 2 if half else 4
    per_step = 2 * 16 + 2 * species + 3 * 4 + 3 * p
    taken = 24 if case["take"] == "device" else 16
    flops = case["steps"] * cells * (2 * case["sweeps"] * 10 + 450)
    return {"bytes": float(cells) * (case["steps"] * per_step + taken), "flops": float(flops)}


# ---- the step in float64 -------------------------------------------------------------------------

MASK64 = (1 << 64) - 1


def _splitmix(v):
    v = (v + 0x9E3779B97F4A7C15) & MASK64
    v = ((v ^ (v >> 30)) * 0xBF58476D1CE4E5B9) & MASK64
    v = ((v ^ (v >> 27)) * 0x94D049BB133111EB) & MASK64
    return v ^ (v >> 31)


def _jitter(seed, frame, amount):
    u = (_splitmix((_splitmix(seed ^ 0xBB67AE8584CAA73B) + frame) & MASK64) >> 40) / 16777216.0
    return 1.0 + amount * (2.0 * u - 1.0)


# the engine's parameter defaults that the step reads
PARAM = dict(burner=3.1, depth=2.7, thickness=1.35, power=2.5, lift=1.6, buoyancy=2.15, persistence=1.45, entrain=1.65,
             fuel=0.30, oxygen=1.0, heat=0.86, vorticity=3.6, domain=(1.15, 1.35, 1.15))
AMBIENT = 300.0


def _shift(f, axis, by):
    """f of the neighbour `by` (-1 or +1) along axis (0 z, 1 y, 2 x), clamped at the walls."""
    n = f.shape[axis]
    if by < 0:
        return torch.cat([f.narrow(axis, 0, 1), f.narrow(axis, 0, n - 1)], axis)
    return torch.cat([f.narrow(axis, 1, n - 1), f.narrow(axis, n - 1, 1)], axis)


def _six(f):
    return sum(_shift(f, a, s) for a in (0, 1, 2) for s in (-1, 1)) / 6.0


def _mix(a, b, t):
    return a * (1.0 - t) + b * t


def _smooth(e0, e1, v):
    t = ((v - e0) / (e1 - e0)).clamp(0.0, 1.0)
    return t * t * (3.0 - 2.0 * t)


class _Exact:
    """One simulation in float64 (the fields as lists of (Z, Y, X) tensors)."""

    def __init__(self, case, dims, seed):
        self.case, self.dims, self.seed = case, dims, seed
        flow, species, pressure = _scene(dims, seed, case["precision"] == "mixed")
        half = case["pressure"] == "f16" or (case["pressure"] == "auto" and math.prod(dims) >= (64 << 20))
        self.flow = [flow[..., c].double() for c in range(4)]
        self.species = [species[..., c].double() for c in range(4)]
        self.p = (pressure.half() if half else pressure).double()
        self.time, self.frame = 0.0, 0
        dev = flow.device
        X, Y, Z = dims
        axis = [torch.arange(n, device=dev, dtype=torch.float64) + 0.5 for n in dims]
        self.px, self.py, self.pz = axis[0].view(1, 1, X), axis[1].view(1, Y, 1), axis[2].view(Z, 1, 1)
        f = lambda v: float(np.float32(v))  # noqa: E731  parameters reach the step as float32
        self.q = {k: (tuple(f(e) for e in v) if isinstance(v, tuple) else f(v)) for k, v in PARAM.items()}
        self.metric = [n / e for n, e in zip(dims, self.q["domain"])]
        self.wall = {}
        for a, (name, n) in enumerate((("z", Z), ("y", Y), ("x", X))):
            i = torch.arange(n, device=dev).view([-1 if k == a else 1 for k in range(3)])
            self.wall[name] = (i == 0, i == n - 1)

    def _advect(self, fields, back):
        X, Y, Z = self.dims
        base, frac = [], []
        for pos, n in zip(back, (X, Y, Z)):
            s = (pos - 0.5).clamp(0.0, float(np.float32(n) - np.float32(1.001)))
            fl = s.floor()
            base.append(fl.long())
            frac.append(s - fl)
        i = base[0] + X * (base[1] + Y * base[2])
        out = []
        for f in fields:
            v = f.reshape(-1)
            z = []
            for oz in (0, X * Y):
                rows = [_mix(v[i + oz + oy], v[i + oz + oy + 1], frac[0]) for oy in (0, X)]
                z.append(_mix(rows[0], rows[1], frac[1]))
            out.append(_mix(z[0], z[1], frac[2]))
        return out

    def _source(self, fuel, temp, power, root):
        q, X, Y, Z = self.q, *self.dims
        thermal = min(root, 1.0 + 0.22 * (root - 1.0))
        if self.case["emitter"] == "spheres":
            j = _jitter(self.seed, self.frame, 0.1)
            source = torch.zeros_like(temp)
            for s in _spheres(self.case, self.dims):
                c, r = [float(np.float32(v)) for v in s["center"]], float(np.float32(s["radius"]))
                d = (self.px - c[0]) ** 2 + (self.py - c[1]) ** 2 + (self.pz - c[2]) ** 2
                inside = d <= r * r
                source = torch.where(inside, torch.ones_like(source), source)
                fuel = torch.where(inside, fuel.clamp(min=s["fuel"] * j), fuel)
                temp = torch.where(inside, temp.clamp(min=AMBIENT + (s["temperature"] - AMBIENT) * j), temp)
            return source, fuel, temp
        ex, ey, ez = q["domain"]
        t = self.time
        x, y, z = self.px / X * ex, self.py / Y * ey, self.pz / Z * ez
        cx, cz = ex * 0.5 + math.sin(t * 1.73) * 0.013, ez * 0.5 + math.cos(t * 1.37) * 0.011
        rx = min(math.sqrt(0.02024) * q["burner"], ex * 0.42)
        rz = min(math.sqrt(0.02024) * q["depth"], ez * 0.42)
        ox, oy, oz = x - cx, y - 0.075, z - cz
        radial = ox * ox / (rx * rx) + oz * oz / (rz * rz)
        vertical = oy * oy / (0.0022 * q["thickness"] ** 2)
        cellular = 0.76 + 0.24 * torch.sin(x * 49.0 + t * 5.2) * torch.sin(z * 43.0 - t * 4.4)
        lobe = torch.sin(ox / rx * 6.2 + t * 1.7) * torch.sin(oz / rz * 5.4 - t * 1.3)
        texture = cellular * _mix(0.48, 1.18, _smooth(-0.42, 0.48, lobe))
        pulse = 0.84 + 0.16 * torch.sin(t * 3.7 + x * 27.0 + z * 21.0)
        source = torch.exp(-(radial + vertical)) * texture * pulse
        return source, torch.maximum(fuel, source * q["fuel"] * power), torch.maximum(temp, AMBIENT + source * 1180.0 * thermal)

    def _simulate(self, dt):
        q, (X, Y, Z), t = self.q, self.dims, self.time
        m = self.metric
        u, v, w, T = self.flow
        flow = self._advect(self.flow + self.species,
                            [self.px - u * dt * m[0], self.py - v * dt * m[1], self.pz - w * dt * m[2]])
        sp = [s.clamp(min=0.0) for s in flow[4:]]
        flow = flow[:4]
        vm, tm, sm = min(dt * 0.32, 0.12), min(dt * 0.18, 0.08), min(dt * 0.12, 0.06)
        flow = [_mix(f, _six(g), tm if c == 3 else vm) for c, (f, g) in enumerate(zip(flow, self.flow))]
        sp = [_mix(f, _six(g), sm) for f, g in zip(sp, self.species)]
        power = q["power"]
        root = math.sqrt(power)
        source, sp[0], flow[3] = self._source(sp[0], flow[3], power, root)
        nx, ny, nz = self.px / X, self.py / Y, self.pz / Z
        s = source * dt * 0.11 * q["vorticity"] * root
        flow[0] = flow[0] + torch.sin(t * 2.3 + nz * 22.0) * s
        flow[2] = flow[2] + torch.cos(t * 1.9 + nx * 25.0) * s
        flow[1] = flow[1] + source * dt * 0.52 * q["lift"] * root
        wall = self.wall
        side = wall["x"][0] | wall["x"][1] | wall["z"][0] | wall["z"][1] | wall["y"][1]
        sp[1] = torch.where(side, sp[1].clamp(min=q["oxygen"]), sp[1])
        flow[3] = torch.where(side, _mix(flow[3], AMBIENT, 0.035), flow[3]).clamp(min=AMBIENT)
        sp[3] = sp[3].clamp(0.0, 3.0)
        o2 = max(q["oxygen"], 0.001)
        deficit = ((o2 - sp[1]) / o2).clamp(0.0, 1.0)
        weight = deficit * _mix(1.0, 0.18, _smooth(0.30, 0.78, sp[0]))
        speed = torch.sqrt(flow[0] ** 2 + flow[1] ** 2 + flow[2] ** 2)
        mix = (dt * q["entrain"] * (0.12 + 0.28 * speed + 0.22 * _smooth(400.0, 1500.0, flow[3])) * weight).clamp(0.0, 0.08)
        sp[1] = _mix(sp[1], o2, mix)
        fuel, oxy = sp[0].clamp(min=0.0), sp[1].clamp(min=0.0)
        available = torch.minimum(fuel, oxy * 0.25)
        rate = (2.5e6 * torch.exp(-15000.0 / flow[3].clamp(min=AMBIENT)) * fuel.clamp(min=1e-5) ** -0.30
                * oxy.clamp(min=1e-5) ** 1.30).clamp(0.0, 80.0)
        burn = available * (1.0 - torch.exp(-rate * _smooth(690.0, 930.0, flow[3]) * dt))
        burn = torch.minimum(burn.clamp(min=0.0), available)
        rich = (1.0 - oxy / (fuel * 4.0).clamp(min=1e-5)).clamp(0.0, 1.0)
        sp[0] = (fuel - burn).clamp(min=0.0)
        sp[1] = (oxy - burn * 4.0).clamp(min=0.0)
        sp[2] = (sp[2] + burn * (1.0 + rich * 1.8)).clamp(0.0, 3.0)
        sp[3] = (sp[3] + burn * 0.62).clamp(0.0, 3.0)
        flow[3] = flow[3] + burn * (2150.0 + 1450.0 * q["heat"])
        reaction = (burn / max(dt, 1e-4) * 0.22).clamp(0.0, 4.0)

        def d(f, a):  # central difference along axis a (0 z, 1 y, 2 x)
            return 0.5 * (_shift(f, a, 1) - _shift(f, a, -1)) * m[2 - a]
        curl = (d(w, 1) - d(v, 0), d(u, 0) - d(w, 2), d(v, 2) - d(u, 1))
        grad = [d(T, 2) + 1e-5, d(T, 1) + 1e-5, d(T, 0) + 1e-5]
        length = torch.sqrt(grad[0] ** 2 + grad[1] ** 2 + grad[2] ** 2)
        grad = [g / length for g in grad]
        vs = 0.00135 * q["vorticity"] * dt
        flow[0] = flow[0] + (grad[1] * curl[2] - grad[2] * curl[1]) * vs
        flow[1] = flow[1] + (grad[2] * curl[0] - grad[0] * curl[2]) * vs
        flow[2] = flow[2] + (grad[0] * curl[1] - grad[1] * curl[0]) * vs
        envelope = _smooth(0.045, 0.15, ny) * (1.0 - _smooth(0.80, 1.0, ny))
        ts = (0.075 + 0.16 * q["vorticity"]) * _smooth(520.0, 1650.0, flow[3]) * envelope * dt
        flow[0] = flow[0] + (torch.sin(ny * 31.0 + nz * 19.0 + t * 3.1) + 0.45 * torch.sin(ny * 67.0 - t * 5.3)) * ts
        flow[1] = flow[1] + 0.12 * torch.sin(nx * 29.0 + nz * 23.0 - t * 4.1) * ts
        flow[2] = flow[2] + (torch.cos(ny * 27.0 - nx * 21.0 + t * 2.7) + 0.45 * torch.cos(ny * 59.0 + t * 4.7)) * ts
        flow[1] = flow[1] + ((flow[3] - AMBIENT) / 1500.0).clamp(-0.1, 1.2) * dt * 0.72 * q["buoyancy"]
        cooling = 5.67e-8 * (AMBIENT ** 4 - flow[3].clamp(min=0.0) ** 4) / (1005.0 * q["persistence"])
        flow[3] = (flow[3] + dt * cooling).clamp(min=AMBIENT)
        out = _smooth(0.84, 0.995, ny)
        decay = torch.exp(-out * dt * 15.0 / q["persistence"])
        sp[2] = sp[2] * math.exp(-dt * 0.075 / q["persistence"]) * decay
        sp[3] = sp[3] * math.exp(-dt * 0.14 / q["persistence"]) * decay
        sp[0] = sp[0] * (1.0 - out)
        flow[3] = _mix(flow[3], AMBIENT, out * 0.16 / q["persistence"])
        reaction = reaction * (1.0 - out)
        top, zero = wall["y"][1], torch.zeros((), dtype=torch.float64, device=u.device)
        for k in (0, 2, 3):
            sp[k] = torch.where(top, zero, sp[k])
        flow[3] = torch.where(top, zero + AMBIENT, flow[3])
        reaction = torch.where(top, zero, reaction)
        flow = self._walls(flow)
        flow = [f.clamp(-1.4, 1.4) if c < 3 else f.clamp(AMBIENT, 2900.0) for c, f in enumerate(flow)]
        return flow, [f.clamp(0.0, 3.0) for f in sp], reaction

    def _walls(self, flow):
        wall, zero = self.wall, torch.zeros((), dtype=torch.float64, device=flow[0].device)
        u = torch.where(wall["x"][0] | wall["x"][1], zero, flow[0])
        w = torch.where(wall["z"][0] | wall["z"][1], zero, flow[2])
        v = torch.where(wall["y"][0], zero, flow[1])
        v = torch.where(wall["y"][1], v.clamp(min=0.0), v)
        return [u, v, w, flow[3]]

    def _divergence(self, flow):
        return sum((flow[c] - _shift(flow[c], 2 - c, -1)) * self.metric[c] for c in range(3))

    def _solve(self, p, div):
        wx, wy, wz = (v * v for v in self.metric)
        for _ in range(self.case["sweeps"]):
            n = wx * (_shift(p, 2, -1) + _shift(p, 2, 1))
            n += wy * (_shift(p, 1, -1) + _shift(p, 1, 1))
            n += wz * (_shift(p, 0, -1) + _shift(p, 0, 1))
            p = (n - div) / (2.0 * (wx + wy + wz))
            p[:, -1, :] = 0.0
        return p

    def _project(self, flow, p):
        grads = [(_shift(p, 2 - c, 1) - p) * self.metric[c] for c in range(3)]
        out = [f - g for f, g in zip(flow, grads)]
        for f in out:
            f[:, -1, :] = f[:, -2, :]  # the open top takes the projected row below
        return self._walls(out + [flow[3]])

    def step(self):
        dt = float(np.float32(DT))
        flow, self.species, self.reaction = self._simulate(dt)
        cold = self.case["pressure"] == "cold"
        self.p = self._solve(torch.zeros_like(self.p) if cold else self.p, self._divergence(flow))
        flow = self._project(flow, self.p)
        correction = self._solve(torch.zeros_like(self.p), self._divergence(flow))
        self.flow = self._project(flow, correction)
        if cold:  # the two solves share their buffers
            self.p = correction
        self.time += DT
        self.frame += 1

    def volumes(self):
        u, v, w, T = self.flow
        s = [f.clamp(min=0.0) for f in self.species]
        reaction = self.reaction.clamp(0.0, 4.0)
        soot = s[2] * _smooth(0.25, 0.82, (s[0] / (s[0] + s[1] * 0.25).clamp(min=0.0001)).clamp(0.0, 1.0))
        shown = torch.maximum(torch.maximum(reaction, soot), torch.maximum(s[3], _smooth(420.0, 700.0, T)))
        return [torch.stack([u, v, w, ((T - 300.0) / 2600.0).clamp(0.0, 1.0)], -1), torch.stack(s, -1),
                torch.stack([reaction, soot, torch.zeros_like(soot), shown], -1)]


def exact(case, seed):
    if case["water"]:  # droplets scatter by a hash of float32 sines: no value in 64 bits
        return None
    dims = _member_dims(case)
    if sum(x * y * z for x, y, z in dims) > EXACT_CELLS:
        return None
    members = []
    for i, d in enumerate(dims):
        e = _Exact(case, d, seed + 101 * i)
        for _ in range(case["steps"]):
            e.step()
        if case["take"] == "device":
            members.append(e.volumes())
            continue
        out = {"flow": torch.stack(e.flow, -1)}
        if case["take"] == "read" and case["steps"] > 1:
            inner = e._divergence(e.flow)[1:-1, 1:-1, 1:-1]
            out |= {"norm": float(inner.square().sum().sqrt()), "largest": float(inner.abs().max())}
        return out
    return members
