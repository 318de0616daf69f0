"""Benchmark cases of the simulation framework.

Each case is one pass that a program makes through the package's public entry
points: a step of a simulation (or of a batch of them) followed by reading the
fields it shows or stores, one stage of the step on its own, a backward pass
of a step, or a rendered frame. The sizes and options are those of the
package's scenes, tests and benchmark, from the smallest domain to the
largest, on both grids and in every storage format.

listed() gives the named cases, draw(rng) another of the same ranges,
prepare(case, seed) the handles and inputs, run(state) one pass, work(case)
the bytes and operations no implementation can avoid, and exact(case, seed)
the outputs in 64 bits where plain torch can give them.
"""
import math

import numpy as np
import torch

from dcgrid_gb300 import Batch, Simulation, capi, scenes
from dcgrid_gb300.sim import default_render_params

PRECISION = {"fp32": capi.PRECISION_FP32, "bf16": capi.PRECISION_MIXED, "fp16": capi.PRECISION_MIXED_FP16}
VELOCITY = ("vel_x", "vel_y", "vel_z")


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the reference application's own scene at its smallest useful size: an
        # interactive frame, where launches and latency count
        dict(name="default_32x64x32", kind="default", gx=32, gy=64, gz=32, blocks=600, iters=10, sphere=False,
             spin=6),
        # the reference's default scene with its sphere obstacle and a converged solve
        dict(name="default_64x128x64_sphere", kind="default", gx=64, gy=128, gz=64, blocks=3000, iters=100,
             sphere=True, spin=6),
        # the pressure projection on its own (stage entry point) of the two-level plume
        dict(name="plume_project_64x128x64", kind="plume_project", gx=64, gy=128, gz=64, levels=2, iters=100,
             spin=6),
        # a three-level plume with FP64 defect correction, bfloat16 scalars, an uneven domain
        dict(name="plume_96x144x80_bf16_defect", kind="plume", gx=96, gy=144, gz=80, levels=3, iters=40,
             precision="bf16", defect=1, spin=6),
        # the terrain cloud at effective 256^3 with a 40000-block budget
        dict(name="cloud_256", kind="cloud", g=256, blocks=40000, levels=3, iters=100, precision="fp32", spin=12),
        # many small simulations at once with the default schedule: parameter studies
        dict(name="batch_10_small", kind="batch", n=10, pick=3, smallest=32, largest=64, iters=20, precision="fp32",
             tuned=False, spin=6),
        # the benchmark's batch: 16 uneven plumes, FP16 scalars, a stored schedule, emission
        # maps from pinned host memory and every member's statistics each step
        dict(name="batch_16_plumes_fp16", kind="batch", n=16, pick=0, smallest=64, largest=256, iters=100,
             precision="fp16", tuned=True, spin=20),
        # the large fire plume: 512^3, four levels allocated in full
        dict(name="fire_512_fp16", kind="fire", g=512, levels=4, iters=100, precision="fp16", spin=2),
        # the uniform grid's step with the reference's sweep counts, an odd-sized domain
        dict(name="uniform_step_150x210x130", kind="uniform_step", gx=150, gy=210, gz=130, iters=10, compat=True),
        # the uniform grid's projection with a converged solve
        dict(name="uniform_project_192", kind="uniform_project", gx=192, gy=192, gz=192, iters=40, compat=False),
        # one step of a reverse sweep through a buoyant rollout: restore, step, adjoint
        dict(name="adjoint_96", kind="adjoint", g=96, levels=2, iters=100, spin=4),
        # a rendered frame of a developed plume, sun shadows on
        dict(name="render_640x360", kind="render", width=640, height=360, g=64, shadows=True, spin=20),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["default", "default", "plume", "plume_project", "cloud", "batch", "batch", "uniform_step",
                       "uniform_project", "adjoint", "render"])
    iters = 2 * round(_log(rng, 5, 50))
    if kind == "default":
        unit = rng.choice([16, 32])  # the derived level count follows from the common power of two
        gx, gy, gz = (unit * max(1, round(_log(rng, 16, 160) / unit)) for _ in range(3))
        full0 = gx * gy * gz // 64
        return dict(kind=kind, gx=gx, gy=gy, gz=gz, blocks=64 + round(full0 * rng.uniform(0.2, 1.1)), iters=iters,
                    sphere=rng.random() < 0.3, spin=4)
    if kind in ("plume", "plume_project"):
        levels = rng.choice([2, 2, 3])
        unit = 4 << (levels - 1)
        gx, gy, gz = (unit * max(2, round(_log(rng, 24, 176) / unit)) for _ in range(3))
        d = dict(kind=kind, gx=gx, gy=gy, gz=gz, levels=levels, iters=iters, spin=4)
        if kind == "plume":
            d.update(precision=rng.choice(["fp32", "bf16", "fp16"]), defect=rng.choice([0, 0, 1]))
        return d
    if kind == "cloud":
        g = 16 * round(_log(rng, 48, 256) / 16)
        return dict(kind=kind, g=g, blocks=round((g // 4) ** 3 * rng.uniform(0.1, 0.4)) + 64, levels=3, iters=iters,
                    precision=rng.choice(["fp32", "bf16", "fp16"]), spin=6)
    if kind == "batch":
        big = rng.random() < 0.4
        return dict(kind=kind, n=rng.randint(2, 18), pick=rng.randint(1, 1000), smallest=32,
                    largest=160 if big else 64, iters=iters, precision=rng.choice(["fp32", "fp16"]),
                    tuned=rng.random() < 0.6, spin=4)
    if kind in ("uniform_step", "uniform_project"):
        gx, gy, gz = (rng.choice([1, 2, 8]) * rng.randint(3, 26) for _ in range(3))
        return dict(kind=kind, gx=max(gx, 17), gy=max(gy, 17), gz=max(gz, 17), iters=iters,
                    compat=rng.random() < 0.4)
    if kind == "adjoint":
        return dict(kind=kind, g=8 * round(_log(rng, 32, 112) / 8), levels=2, iters=iters, spin=3)
    return dict(kind="render", width=round(_log(rng, 100, 900)), height=round(_log(rng, 80, 600)),
                g=rng.choice([32, 64, 96]), shadows=rng.random() < 0.5, spin=10)


# ------------------------------------------------------------------ parameters
def _params(c):
    """The simulation parameters of a case (a list of them for a batch)."""
    k = c["kind"]
    if k == "default":
        p = scenes.ref_default(c["gx"], c["gy"], c["gz"], c["blocks"],
                               capi.SOLIDS_SPHERE if c["sphere"] else capi.SOLIDS_NONE)
        p.jacobi_iters = c["iters"]
        return p
    if k in ("plume", "plume_project"):
        p = scenes.plume(c["gx"], c["gy"], c["gz"], _half_budget(c), c["levels"], c["iters"])
        p.precision = PRECISION[c.get("precision", "fp32")]
        p.defect_passes = c.get("defect", 0)
        return p
    if k == "cloud":
        p = scenes.cloud(c["g"], c["blocks"], c["levels"], c["iters"])
        p.terrain_amplitude = 40.0 * c["g"] / 256.0
        p.terrain_base_height = 8.0 * c["g"] / 256.0
        p.precision = PRECISION[c["precision"]]
        p.emission_n = 16
        p.emission_band = 16.0
        return p
    if k == "fire":
        return scenes.fire(c["g"], c["levels"], PRECISION[c["precision"]], 100 * 10 ** 9, c["iters"])
    if k == "batch":
        sizes = [s for s in (32, 48, 64, 96, 128, 160, 192, 256) if c["smallest"] <= s <= c["largest"]]
        if c["largest"] == 256:
            sizes = [64, 96, 128, 192, 256]
        return scenes.plume_batch(c["n"], c["pick"], tuple(sizes), c["iters"], PRECISION[c["precision"]],
                                  em_n=16)
    if k in ("uniform_step", "uniform_project"):
        p = capi.default_params(c["gx"], c["gy"], c["gz"], 0)
        p.jacobi_iters = c["iters"]
        p.ref_compat = 1 if c["compat"] else 0
        return p
    if k == "adjoint":
        p = scenes.differentiable(c["g"], c["levels"], c["iters"])
        p.n_scalars = 3
        p.buoy_alpha, p.buoy_beta = 0.1, 0.3
        p.src_enabled = 1
        p.src_center[0] = p.src_center[2] = c["g"] / 2.0
        p.src_center[1] = c["g"] / 8.0
        p.src_radius = c["g"] / 12.0
        p.src_density, p.src_temperature = 1.0, 2.0
        return p
    p = scenes.plume(c["g"], 2 * c["g"], c["g"], None, 2, 20)
    p.src_radius = c["g"] / 6.0
    p.src_center[1] = c["g"] / 4.0
    return p


def _half_budget(c):
    """Coarser levels in full and half of the finest."""
    full = [(c["gx"] >> (l + 2)) * (c["gy"] >> (l + 2)) * (c["gz"] >> (l + 2)) for l in range(c["levels"])]
    return sum(full[1:]) * 3 // 2 + full[0] // 2


def _tuning(batch):
    """The schedule that a program stored after it had tuned such a batch once."""
    t = batch.get_tuning()
    for i in range(4):
        t.tile[i] = 1
    t.persistent = 1
    t.solve_cache = 19
    t.solve_ctas_per_sm = 0
    t.solve_barrier = 3
    return t


def _noise(shape, seed, amplitude, cells=12):
    """Smooth random field: white noise on a coarse lattice, interpolated."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    low = [max(2, n // cells) for n in shape]
    f = torch.rand([1, 1] + low, generator=gen, device="cuda") * 2 - 1
    f = torch.nn.functional.interpolate(f, size=tuple(shape), mode="trilinear", align_corners=True)
    return (amplitude * f[0, 0]).contiguous()


def prepare(case, seed):
    k = case["kind"]
    p = _params(case)
    if k == "batch":
        b = Batch(p)
        if case["tuned"]:
            b.set_tuning(_tuning(b))
        rng = np.random.default_rng(seed)
        n = sum(q.emission_n ** 3 for q in p)
        maps = torch.from_numpy((0.05 * rng.random(n)).astype(np.float32)).pin_memory()
        b.set_emission(maps)
        for i, m in enumerate(b.members):
            m.add_velocity_noise(seed + i, 0.05 * m.params.dx / m.params.dt)
        b.step(case["spin"])
        b.sync()
        out = [torch.empty(m.num_cells, device="cuda") for m in b.members]
        return dict(case=case, batch=b, maps=maps, out=out)
    if k in ("uniform_step", "uniform_project"):
        s = Simulation(p, capi.MODE_UNIFORM)
        shape = (p.gz, p.gy, p.gx)
        for i, f in enumerate(VELOCITY):
            s.set_field(f, _noise(shape, 8 * seed + i, 1.5 * p.dx / p.dt).reshape(-1))
        s.set_field("density", (_noise(shape, 8 * seed + 3, 1.0).abs()).reshape(-1))
        names = VELOCITY + (("density", "pressure") if k == "uniform_step" else ("pressure", "divergence"))
        return dict(case=case, sim=s, out={f: torch.empty(s.num_cells, device="cuda") for f in names})
    s = Simulation(p, capi.MODE_ADAPTIVE)
    if p.emission_n > 0:
        s.set_emission(scenes.emission_field(p.emission_n, seed))
    s.add_velocity_noise(seed, 0.05 * p.dx / p.dt)
    if case["spin"]:
        s.step(case["spin"])
    s.sync()
    state = dict(case=case, sim=s)
    if k == "adjoint":
        stream = torch.cuda.Stream()
        s.set_stream(stream.cuda_stream)
        before = torch.empty(s.state_bytes(), dtype=torch.uint8, device="cuda")
        s.save_state(before)
        gen = torch.Generator(device="cuda").manual_seed(seed)
        n = (3 + p.n_scalars) * s.num_cells
        lam = torch.randn(n, generator=gen, device="cuda")
        torch.cuda.synchronize()
        state.update(stream=stream, before=before, lam=lam, lam_out=torch.empty(n, device="cuda"),
                     lam_em=torch.empty(p.emission_n ** 3, device="cuda"),
                     density=torch.empty(s.num_cells, device="cuda"))
    elif k == "render":
        rp = default_render_params(case["width"], case["height"], p)
        rp.shadows = 1 if case["shadows"] else 0
        state.update(rp=rp, image=torch.empty((case["height"], case["width"], 4), device="cuda"))
    else:
        names = VELOCITY + (("pressure", "divergence") if k == "plume_project" else ("density", "pressure"))
        if k == "fire":
            names = ("density", "vel_y")
        state["out"] = {f: torch.empty(s.num_cells, device="cuda") for f in names}
    return state


def run(state):
    k = state["case"]["kind"]
    if k == "batch":
        b = state["batch"]
        b.set_emission(state["maps"])
        b.step(1)
        stats = b.stats()
        for m, o in zip(b.members, state["out"]):
            m.get_field("density", out=o)
        return dict(density=state["out"], mass=np.array([st.mass for st in stats]),
                    residual=np.array([st.residual for st in stats]),
                    cells=np.array([st.active_cells for st in stats]))
    s = state["sim"]
    if k == "adjoint":
        with torch.cuda.stream(state["stream"]):
            s.load_state(state["before"])
            state["lam_em"].zero_()
            s.adjoint_step_full(state["lam"], state["lam_out"], state["lam_em"])
            s.get_field("density", out=state["density"])
        return dict(lam=state["lam_out"], emission=state["lam_em"], density=state["density"])
    if k == "render":
        return s.render(state["rp"], out=state["image"])
    if k in ("plume_project", "uniform_project"):
        s.project()
    else:
        s.step(1)
    for f, o in state["out"].items():
        s.get_field(f, out=o)
    return state["out"]


# ------------------------------------------------------------------ floors
def _cells(p, fill):
    """Cells of every level under the block budget; levels that the budget does
    not cover in full count with the share `fill`."""
    levels = p.levels
    if levels == 0:
        levels, size = 1, 2
        small = min(p.gx, p.gy, p.gz)
        while p.gx % size == 0 and p.gy % size == 0 and p.gz % size == 0 and size * 4 <= small:
            levels += 1
            size *= 2
    full = [(p.gx >> (l + 2)) * (p.gy >> (l + 2)) * (p.gz >> (l + 2)) for l in range(levels)]
    cells, left = 64.0 * full[-1], p.max_blocks - full[-1]
    for l in range(levels - 2, -1, -1):
        take = min(left // (l + 1), full[l])
        left -= take
        cells += 64.0 * take * (1.0 if take == full[l] else fill)
    return cells


def work(case):
    k = case["kind"]
    p = _params(case)
    if k == "render":
        pixels = case["width"] * case["height"]
        cells = _cells(p, 1.0)
        return {"bytes": 16.0 * pixels + 4.0 * cells, "flops": 30.0 * pixels * 2 * p.gz}
    if k in ("uniform_step", "uniform_project"):
        cells = float(p.gx) * p.gy * p.gz
        sweeps = 2.0 if case["compat"] else float(case["iters"])
        step = k == "uniform_step"
        # velocity, fluidity (and density) in, velocity, pressure (and density or divergence) out
        return {"bytes": cells * (4 * 4 + 4 * 5 + (4 if step else 0)),
                "flops": cells * (8 / 7 * 8 * sweeps + (250 if step else 40))}
    members = p if k == "batch" else [p]
    total = {"bytes": 0.0, "flops": 0.0}
    for q in members:
        cells = _cells(q, 0.3 if k in ("batch", "plume", "plume_project") else 1.0)
        sq = 4 if q.precision == capi.PRECISION_FP32 else 2
        if k == "plume_project":
            total["bytes"] += cells * (4 * 4 + 4 * 5)
            total["flops"] += cells * (8 * q.jacobi_iters + 40)
        elif k == "adjoint":
            # state and adjoint in, state and adjoint out
            total["bytes"] += cells * 4 * (4 + 3 + 6 + 4 + 3 + 6)
            total["flops"] += cells * (16 * q.jacobi_iters + 900)
        else:
            total["bytes"] += cells * (4 * 4 + 4 * 4 + 2 * sq * q.n_scalars)
            total["flops"] += cells * (8 * q.jacobi_iters * (1 + q.defect_passes) + 350)
    return total


# ------------------------------------------------------------------ 64-bit values
def exact(case, seed):
    if case["kind"] == "plume_project":
        return _exact_adaptive_project(case, seed)
    if case["kind"] in ("uniform_step", "uniform_project"):
        return _exact_uniform(case, seed)
    return None  # topology decisions and scattered samples: no plain 64-bit form


def _exact_uniform(case, seed):
    s = prepare(case, seed)["sim"]
    p = s.params
    shape = (p.gz, p.gy, p.gx)

    def field(name):
        t = torch.empty(s.num_cells, device="cuda")
        s.get_field(name, out=t)
        return t.double().reshape(shape)

    vel = [field(f) for f in VELOCITY]
    density = field("density")
    rdx = float(np.float32(1.0) / np.float32(p.dx))
    dt, dx = float(p.dt), float(p.dx)
    z, y, x = torch.meshgrid(*(torch.arange(-1, n + 1, device="cuda", dtype=torch.float64) for n in shape),
                             indexing="ij")
    inlet = (y < 0) & (torch.sqrt((x - 0.5 * p.gx) ** 2 + (z - 0.5 * p.gz) ** 2) < p.emission_radius * rdx)
    if not p.inlet_enabled:
        inlet = torch.zeros_like(inlet)

    def padded(f, at_inlet):
        # one layer of boundary values around the domain: closed walls and the inlet
        g = torch.nn.functional.pad(f, (1, 1, 1, 1, 1, 1))
        return torch.where(inlet, torch.full_like(g, at_inlet), g)

    at = (0.0, float(p.velocity_emission_rate), 0.0)

    def sample(pads, v):
        zc, yc, xc = torch.meshgrid(*(torch.arange(n, device="cuda", dtype=torch.float64) for n in shape),
                                    indexing="ij")
        pos = [xc - v[0] * dt * rdx, yc - v[1] * dt * rdx, zc - v[2] * dt * rdx]
        low = [torch.floor(q) for q in pos]
        frac = [q - l for q, l in zip(pos, low)]
        out = [torch.zeros_like(xc) for _ in pads]
        dims = (p.gx, p.gy, p.gz)
        for c in range(8):
            bit = ((c >> 2) & 1, (c >> 1) & 1, c & 1)
            i = [((l + b).clamp(-1, n) + 1).long() for l, b, n in zip(low, bit, dims)]
            w = torch.ones_like(xc)
            for f, b in zip(frac, bit):
                w = w * (f if b else 1 - f)
            for o, g in zip(out, pads):
                o += w * g[i[2], i[1], i[0]]
        return out

    step = case["kind"] == "uniform_step"
    if step:
        vel = sample([padded(f, a) for f, a in zip(vel, at)], vel)
    px, py, pz = (padded(f, a) for f, a in zip(vel, at))
    div = 0.5 * rdx * (px[1:-1, 1:-1, 2:] - px[1:-1, 1:-1, :-2] + py[1:-1, 2:, 1:-1] - py[1:-1, :-2, 1:-1] +
                       pz[2:, 1:-1, 1:-1] - pz[:-2, 1:-1, 1:-1])
    divs, size, small = [div], 2, min(p.gx, p.gy, p.gz)
    while p.gx % size == 0 and p.gy % size == 0 and p.gz % size == 0 and size * 4 <= small:
        d = divs[-1]
        divs.append(0.125 * sum(d[a::2, b::2, c::2] for a in (0, 1) for b in (0, 1) for c in (0, 1)))
        size *= 2

    def neighbours(f):
        g = torch.nn.functional.pad(f[None, None], (1,) * 6, mode="replicate")[0, 0]
        return (g[1:-1, 1:-1, :-2], g[1:-1, 1:-1, 2:], g[1:-1, :-2, 1:-1], g[1:-1, 2:, 1:-1], g[:-2, 1:-1, 1:-1],
                g[2:, 1:-1, 1:-1])

    def prolong(c):
        def axis(n):
            i = torch.arange(2 * n, device="cuda")
            s = torch.where((i == 0) | (i == 2 * n - 1), 0, 2 * (i % 2) - 1)
            return i // 2, i // 2 + s
        (z0, z1), (y0, y1), (x0, x1) = (axis(n) for n in c.shape)

        def at3(a, b, d):
            return c[a][:, b][:, :, d]
        return (27 * at3(z0, y0, x0) + 9 * (at3(z0, y0, x1) + at3(z0, y1, x0) + at3(z1, y0, x0)) +
                3 * (at3(z0, y1, x1) + at3(z1, y0, x1) + at3(z1, y1, x0)) + at3(z1, y1, x1)) / 64

    pr = torch.zeros_like(divs[-1])
    for l in range(len(divs) - 1, -1, -1):
        if l < len(divs) - 1:
            pr = prolong(pr)
        pairs = (2 if l == len(divs) - 1 else 1) if case["compat"] else case["iters"] // 2
        for _ in range(2 * pairs):
            pr = (sum(neighbours(pr)) - (dx * 2 ** l) ** 2 * divs[l]) / 6
    n = neighbours(pr)
    vel = [v - 0.5 * rdx * (n[2 * a + 1] - n[2 * a]) for a, v in enumerate(vel)]
    out = dict(zip(VELOCITY, (v.reshape(-1) for v in vel)))
    out["pressure"] = pr.reshape(-1)
    if step:
        out["density"] = sample([padded(density, float(p.density_emission_rate))], vel)[0].reshape(-1)
    else:
        out["divergence"] = div.reshape(-1)
    return out


def _exact_adaptive_project(case, seed):
    s = prepare(case, seed)["sim"]
    p = s.params
    topo = s.get_topology()
    pos = torch.from_numpy(topo["pos"]).cuda().long()
    parent = torch.from_numpy(topo["parent"].astype(np.int64)).cuda()
    none = 0xFFFFFFFF
    child = torch.from_numpy(topo["child"].astype(np.int64)).cuda()
    apron = torch.from_numpy(s.get_apron()).cuda().reshape(-1, 6, 6, 6)
    nc = s.num_cells

    def field(name):
        t = torch.empty(nc, device="cuda")
        s.get_field(name, out=t)
        return t.double()

    vel = [field(f) for f in VELOCITY]
    w = field("fluidity")
    c = torch.arange(64, device="cuda")
    local = [2 * ((c >> (5 - a)) & 1) + ((c >> (2 - a)) & 1) for a in range(3)]  # x, y, z of a cell in its block
    faces = [(-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1)]
    near = torch.stack([apron[:, local[0] + 1 + d[0], local[1] + 1 + d[1], local[2] + 1 + d[2]] for d in faces], -1)
    level = pos[:, 3]
    scale = (2.0 ** level.clamp(min=0).double())[:, None]
    rdx = float(np.float32(1.0) / np.float32(p.dx))
    dims = (p.gx, p.gy, p.gz)
    leaf = ((child == none) & (level >= 0)[:, None]).repeat_interleave(8, dim=1)
    div = torch.zeros((pos.shape[0], 64), dtype=torch.float64, device="cuda")
    safe = near.clamp(min=0)
    for f, d in enumerate(faces):
        a = f // 2
        q = (pos[:, a, None] + local[a] + d[a]) * scale
        inside = (q >= 0) & (q < dims[a])
        term = torch.where(inside, w[safe[..., f]] * vel[a][safe[..., f]], 0.0)
        div += (1 if f % 2 else -1) * 0.5 * rdx / scale * term
    div = torch.where(leaf, div, 0.0).reshape(-1)
    blocks = [torch.nonzero(level == l).reshape(-1) for l in range(int(level.max()) + 1)]

    def restrict(f):
        for l in range(len(blocks) - 1):
            b = blocks[l]
            mean = f.reshape(-1, 8, 8)[b].mean(-1)
            par = parent[b]
            f.reshape(-1, 8, 8)[par // 8, par % 8] = mean
        return f

    div = restrict(div)
    plane = [torch.zeros(nc, dtype=torch.float64, device="cuda") for _ in range(2)]
    for l in range(len(blocks) - 1, -1, -1):
        b = blocks[l]
        cells = (64 * b[:, None] + c).reshape(-1)
        at = near[b].reshape(-1, 6)
        if l < len(blocks) - 1:
            ap = apron[parent[b] // 8]
            g = [pos[b, a, None] + local[a] for a in range(3)]
            base = [1 + (q // 2) % 4 for q in g]
            side = [q % 2 * 2 - 1 for q in g]
            row = torch.arange(len(b), device="cuda")[:, None]
            value = 0
            for m in range(8):
                bit = ((m >> 2) & 1, (m >> 1) & 1, m & 1)
                i = [q + e * t for q, e, t in zip(base, side, bit)]
                value = value + (27, 9, 3, 1)[sum(bit)] * plane[0][ap[row, i[0], i[1], i[2]]]
            plane[0][cells] = (value / 64).reshape(-1)
        alpha = float(p.dx) ** 2 * 4.0 ** l
        for it in range(case["iters"]):
            plane[(it + 1) & 1][cells] = (plane[it & 1][at].sum(-1) - alpha * div[cells]) / 6
    pr = plane[0]
    for a in range(3):
        lo, hi = safe[..., 2 * a], safe[..., 2 * a + 1]
        pc = pr.reshape(-1, 64)
        dv = 0.5 * rdx / scale * (w[hi] * (pr[hi] - pc) + w[lo] * (pc - pr[lo]))
        v = vel[a].reshape(-1, 64)
        vel[a] = restrict(torch.where(leaf, v - dv, v).reshape(-1).clone())
    out = dict(zip(VELOCITY, vel))
    out["pressure"] = pr
    out["divergence"] = div
    return out
