"""What users of gargantua_b200 have it do, as measurable cases: stills and
streams of stills through the server, live frames (step, splat, march, tone
curve), the splat of a whole disk into sums that ranks combine, settling and
reading a particle system, baked frames, probe rays.

Sizes are the presets' (cli.PRESETS), the request stream's of bench.py and
odd ones around them. Every input comes from the seed: cameras, star seeds,
particles and the gas volume.

`exact` renders the same rays in float64 with torch (RK4 with the same step
policy, trilinear gas, starfield), and steps particles in float64, without
the library.
"""
import math
import random

import numpy as np
import torch

import gargantua_b200 as g
from gargantua_b200 import parallel
from gargantua_b200 import types as T

# The request stream of bench.py.
RESOLUTIONS = [(320, 180), (640, 360), (960, 540), (1920, 1080), (3840, 2160)]
SPINS = [0.0, 0.5, 0.9]
BUDGET = 24 << 30  # a server-sized memory budget, as bench.py gives its context


def listed():
    return [
        # A validation program's camera grid of rays: the smallest call, one ray's latency.
        {"name": "probes_kerr_8x8", "kind": "probes", "columns": 8, "rows": 8, "spin": 0.9},
        # One preview request, as an interactive client sends: launches, copies and the scheduler's own time.
        {"name": "request_320x180", "kind": "serve", "count": 1, "width": 320, "height": 180, "cap": 256, "spin": 0.0},
        # A burst of small previews and thumbnails of several clients.
        {"name": "burst_small", "kind": "serve", "count": 24, "width": 0, "height": 360, "cap": 0, "spin": -1.0},
        # The still of the command line (4096 steps), without and with spin.
        {"name": "still_1920x1080", "kind": "serve", "count": 1, "width": 1920, "height": 1080, "cap": 4096, "spin": 0.0},
        {"name": "still_kerr_1920x1080", "kind": "serve", "count": 1, "width": 1920, "height": 1080, "cap": 4096, "spin": 0.9},
        # A slice of the served request stream, all sizes, step budgets and spins.
        {"name": "stream_mixed", "kind": "serve", "count": 12, "width": 0, "height": 2160, "cap": 0, "spin": -1.0},
        # A served sequence frame of the default preset: step, stochastic splat, interactive request.
        {"name": "sequence_default", "kind": "sequence", "particles": 1_000_000, "volume": 128, "width": 960, "height": 540, "spin": 0.0},
        # A live frame of the max preset: step, exact splat, per-request march, tone curve.
        {"name": "frame_max", "kind": "frame", "particles": 4_000_000, "volume": 256, "width": 960, "height": 540, "exact": True, "spin": 0.0},
        # A live Kerr frame of the small preset in an odd window.
        {"name": "frame_small_kerr", "kind": "frame", "particles": 250_000, "volume": 96, "width": 1001, "height": 563, "exact": False, "spin": 0.5},
        # The max preset's particles binned into sums that ranks then add up.
        {"name": "bin_exact_max", "kind": "bin", "particles": 4_000_000, "volume": 256, "exact": True},
        # Settling a default disk and taking its state (checkpoints, checksums).
        {"name": "settle_default", "kind": "settle", "particles": 1_000_000, "dispatches": 300},
        # The bake strategy's frame for a new camera: bake, walk, tone curve.
        {"name": "bake_960x540", "kind": "bake", "volume": 128, "width": 960, "height": 540},
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["probes", "serve", "serve", "serve", "sequence", "frame", "bin", "settle", "bake"])
    spin = rng.choice(SPINS)
    size = {"width": log(161, 1920), "height": log(91, 1080)}
    disk = {"particles": log(50_000, 4_000_000), "volume": rng.choice([96, 100, 128, 192, 256])}
    if kind == "probes":
        return {"kind": kind, "columns": log(2, 9), "rows": log(2, 9), "spin": spin}
    if kind == "serve":
        count = log(1, 12)
        if count > 4:
            return {"kind": kind, "count": count, "width": 0, "height": rng.choice([360, 540, 1080]), "cap": 0, "spin": -1.0, "mix": rng.randrange(1 << 20)}
        return {"kind": kind, "count": count, **size, "cap": rng.choice([256, 4096]), "spin": spin}
    if kind == "sequence":
        return {"kind": kind, **disk, **size, "spin": spin}
    if kind == "frame":
        return {"kind": kind, **disk, **size, "exact": rng.random() < 0.5, "spin": spin}
    if kind == "bin":
        return {"kind": kind, **disk, "exact": rng.random() < 0.7}
    if kind == "settle":
        return {"kind": kind, "particles": log(1000, 1_000_000), "dispatches": log(1, 300)}
    return {"kind": kind, "volume": disk["volume"], "width": min(size["width"], 960), "height": min(size["height"], 540)}


# ------------------------------------------------------------------ inputs


def requests(case, seed=0):
    """A serve case's requests: sizes, budgets and spins from the case, cameras and stars from the seed."""
    mix, rng = random.Random(case.get("mix", 7)), random.Random(seed)
    out = []
    for k in range(case["count"]):
        w, h = case["width"], case["height"]
        if w == 0:  # every resolution up to the case's height, in turn
            sizes = [r for r in RESOLUTIONS if r[1] <= h]
            w, h = sizes[(len(sizes) - 1 - k) % len(sizes)]
        cap = case["cap"] or mix.choice([256, 4096])
        spin = case["spin"] if case["spin"] >= 0.0 else mix.choice(SPINS)
        out.append({"width": w, "height": h, "cap": cap, "spin": spin, "azimuth": rng.uniform(0.0, 2.0 * math.pi),
                    "elevation": math.pi / 2.0 - math.radians(rng.uniform(30.0, 88.0)), "distance": rng.uniform(42.0, 70.0),
                    "stars": rng.randrange(1 << 32)})
    return out


def gas(size, seed, device):
    """A settled disk's two textures (half4 emission and density, half4 velocity), float16 (n^3, 4): 1M particles
    between the innermost stable orbit and r = 24, thickness 0.05 r, counted per voxel."""
    gen = torch.Generator(device=device).manual_seed(seed & 0x7FFFFFFF)
    n, count = size, 1_000_000

    def rand():
        return torch.rand(count, generator=gen, device=device, dtype=torch.float64)

    r = 6.0 + 18.0 * rand() ** 0.8
    phi = 2.0 * math.pi * rand()
    z = 0.05 * r * torch.randn(count, generator=gen, device=device, dtype=torch.float64)
    p = torch.stack([r * torch.cos(phi), r * torch.sin(phi), z], 1)
    i = ((p + 30.0) / 60.0 * n).floor().long().clamp_(0, n - 1)
    cell = (i[:, 2] * n + i[:, 1]) * n + i[:, 0]
    mass = torch.bincount(cell, minlength=n**3).double()
    # Four sums per voxel; a fixed-point sum is the same whatever order the adds take.
    t4 = (6.0 / r) ** 3 * (1.0 - torch.sqrt(6.0 / r)).clamp_min(0.01) / 0.057
    v = torch.sqrt(r) / (r - 2.0)
    sums = torch.zeros(n**3, 3, device=device, dtype=torch.int64)
    words = torch.stack([t4, -v * torch.sin(phi), v * torch.cos(phi)], 1)
    sums.index_add_(0, cell, (words * 65536.0).round().long())
    sums = sums.double() / 65536.0
    inv = (n / 60.0) ** 3
    e = torch.zeros(n**3, 4, device=device, dtype=torch.float64)
    warm = torch.tensor([1.0, 0.86, 0.72], device=device, dtype=torch.float64)
    e[:, :3] = sums[:, :1] * warm * 5e-4 * inv
    e[:, 3] = mass * inv
    u = torch.zeros_like(e)
    u[:, :2] = sums[:, 1:] / mass.clamp_min(1.0)[:, None]
    u[:, 3] = 1.0
    return e.half(), u.half()


def particles(count, seed):
    """Particle records (position, velocity, temperature, respawns as bits) of a disk in motion."""
    rng = np.random.default_rng(seed)
    r = 6.0 + 18.0 * rng.random(count) ** 0.8
    phi = 2.0 * math.pi * rng.random(count)
    vc = np.sqrt(r) / (r - 2.0)
    noise = 0.02 * vc[:, None] * rng.standard_normal((count, 3))
    out = np.zeros((count, 8), np.float32)
    out[:, 0], out[:, 1], out[:, 2] = r * np.cos(phi), r * np.sin(phi), 0.05 * r * rng.standard_normal(count)
    out[:, 3:6] = np.stack([-vc * np.sin(phi), vc * np.cos(phi), 0.0 * vc], 1) + noise
    out[:, 6] = 8000.0 * (6.0 / r) ** 0.75
    return out


def camera(seed):
    rng = random.Random(seed)
    return g.OrbitCamera(rng.uniform(0.0, 2.0 * math.pi), rng.uniform(0.05, 0.9), rng.uniform(45.0, 58.0))


def device_of():
    return "cuda" if torch.cuda.is_available() else "cpu"


def prepare(case, seed):
    kind = case["kind"]
    ctx = g.Context(0, budget_bytes=BUDGET)
    s = {"case": case, "ctx": ctx}
    if kind == "probes":
        s["launches"] = g.camera_grid(camera(seed), case["columns"], case["rows"], 16 / 9)
        s["u"] = g.uniforms(camera(seed), 1, 1, g.Settings.still(), 1e-5, False, 0, spin=case["spin"])
        return s
    if kind == "serve":
        s["volume"] = g.Volume(ctx, 128)
        e, v = gas(128, seed, device_of())
        s["volume"].write(e.cpu().numpy(), v.cpu().numpy())
        s["specs"] = [g.RequestSpec(q["width"], q["height"], q["cap"], q["spin"], q["azimuth"], q["elevation"], q["distance"],
                                    star_seed=q["stars"]) for q in requests(case, seed)]
        s["outputs"] = [g.pinned_array(ctx, (q.width * q.height, 4), np.float16) for q in s["specs"]]
        s["server"] = g.Server(ctx, s["volume"])
        return s
    if kind == "sequence":
        s["server"] = g.Server(ctx, None)
        s["sequence"] = g.Sequence(s["server"], ctx, case["particles"], case["volume"], 1 << 30, case["width"], case["height"],
                                   case["spin"], seed & 0xFFFFFFFF, camera(seed), settle_dispatches=40)
        return s
    if kind == "bake":
        s["volume"] = g.Volume(ctx, case["volume"])
        e, v = gas(case["volume"], seed, device_of())
        s["volume"].write(e.cpu().numpy(), v.cpu().numpy())
    else:
        s["particles"] = g.Particles(ctx, case["particles"], seed)
        if kind == "settle":
            s["particles"].write(particles(case["particles"], seed))
            return s
        s["particles"].advance(100, seed_first=True)
        s["volume"] = g.Volume(ctx, case["volume"])
        if kind == "bin":
            s["sums"] = parallel.device_sums(s["volume"])
            s["sums"].owner = s["volume"]  # the tensor aliases the volume's memory, so it keeps the volume
            return s
    cam = camera(seed)
    s["targets"] = g.Targets(ctx, case["width"], case["height"])
    s["u"] = g.uniforms(cam, case["width"], case["height"], g.Settings.interactive(), 1e-4, True, seed & 0xFFFFFFFF,
                        spin=case.get("spin", 0.0), bake_spacing=g.Bake.spacing(case["volume"]) if kind == "bake" else 0.0)
    if case.get("spin", 0.0) == 0.0:
        ctx.enable_tables(s["u"], float(np.float32(cam.distance)))
    if kind == "bake":
        s["bake"] = g.Bake(ctx, case["width"], case["height"])
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "probes":
        r = s["ctx"].probe(s["launches"], s["u"], T.PRECISION_COMPENSATED)
        return {"position": r["position"], "direction": r["direction"]}
    if kind == "serve":
        server = s["server"]
        tickets = [server.submit(q, o) for q, o in zip(s["specs"], s["outputs"])]
        return [server.wait(t)[0] for t in tickets]
    if kind == "sequence":
        return s["sequence"].frame()[0]
    if kind == "frame":
        s["particles"].step(1)
        s["volume"].splat(s["particles"], exact=case["exact"])
        g.march(s["ctx"], s["volume"], s["u"], s["targets"])
        return s["targets"].tonemap()
    if kind == "bin":
        s["volume"].clear()
        s["volume"].bin(s["particles"], case["exact"])
        return s["sums"]
    if kind == "settle":
        s["particles"].step(case["dispatches"])
        r = s["particles"].read()
        return {"state": r[:, :7], "respawns": r[:, 7].view(np.uint32)}
    s["bake"].bake_full(s["u"])
    s["bake"].walk(s["volume"], s["u"], s["targets"])
    return s["targets"].tonemap()


# What a ray takes: RK4 steps a ray of these cameras (measured with the library's own counters) and the floating
# point operations of one (oracle/opcount.cpp): Kerr 515, Schwarzschild 192 and 111 for each sample in the slab.
STEPS = {(True, 256): 215, (True, 4096): 235, (False, 256): 30, (False, 4096): 58}


def march_flops(rays, spin, cap):
    steps = rays * STEPS[(spin > 0.0, cap)]
    return steps * (515.0 if spin > 0.0 else 192.0 + 30.0)


def work(case):
    kind = case["kind"]
    if kind == "probes":
        n = case["columns"] * case["rows"]
        return {"bytes": n * 68.0, "flops": march_flops(n, case["spin"], 4096)}
    if kind == "serve":
        q = requests(case)
        return {"bytes": 16.0 * 128**3 + sum(8.0 * r["width"] * r["height"] for r in q),
                "flops": sum(march_flops(r["width"] * r["height"], r["spin"], r["cap"]) for r in q)}
    if kind == "settle":
        # State in and out once; two substeps of about 60 operations a dispatch.
        return {"bytes": 64.0 * case["particles"], "flops": 120.0 * case["particles"] * case["dispatches"]}
    if kind == "bin":
        # Particles read, 24-byte records written once; 48 values of 3 operations for an exact deposit.
        return {"bytes": 32.0 * case["particles"] + 24.0 * case["volume"] ** 3,
                "flops": case["particles"] * (20.0 + (144.0 if case["exact"] else 18.0))}
    px = float(case["width"] * case["height"])
    if kind == "bake":
        return {"bytes": 4.0 * px + 16.0 * case["volume"] ** 3, "flops": march_flops(px, 0.0, 256)}
    splat = 64.0 * case["particles"] + 16.0 * case["volume"] ** 3
    out = 4.0 if kind == "frame" else 8.0
    return {"bytes": splat + out * px, "flops": march_flops(px, case["spin"], 256) + 120.0 * case["particles"]}


# ------------------------------------------------- the same in 64 bits

F = torch.float64
SLAB, HALF, CAPTURE = 6.0, 30.0, float(np.float32(2.02))


def f32(x):
    return float(np.float32(x))


def basis(azimuth, elevation, distance):
    az, el, d = f32(azimuth), f32(elevation), f32(distance)
    pos = d * np.array([math.cos(el) * math.cos(az), math.cos(el) * math.sin(az), math.sin(el)])
    fwd = -pos / np.linalg.norm(pos)
    right = np.cross(fwd, [0.0, 0.0, 1.0])
    right /= np.linalg.norm(right)
    return pos, right, np.cross(right, fwd), fwd


def unit(v):
    return v / v.norm(dim=1, keepdim=True)


def camera_rays(q, device):
    pos, right, up, fwd = basis(q["azimuth"], q["elevation"], q["distance"])
    t = math.tan(0.5 * f32(50.0 * math.pi / 180.0))
    w, h = q["width"], q["height"]
    x = (2.0 * (torch.arange(w, device=device, dtype=F) + 0.5) / w - 1.0) * t * w / h
    y = (1.0 - 2.0 * (torch.arange(h, device=device, dtype=F) + 0.5) / h) * t
    right, up, fwd = (torch.tensor(v, device=device, dtype=F) for v in (right, up, fwd))
    d = fwd + x[None, :, None] * right + y[:, None, None] * up
    return torch.tensor(pos, device=device, dtype=F).expand(w * h, 3), unit(d.reshape(-1, 3))


def settings(cap):
    """The step policy of a request: interactive up to 256 steps, else the still's."""
    return {"cap": cap, "empty": f32(0.1) if cap <= 256 else f32(0.06), "empty_max": 3.0 if cap <= 256 else 1.5}


def sweep(r, b, nodes=400):
    """Azimuth from radius r to infinity of a ray of impact parameter b."""
    bmax = r / torch.sqrt(1.0 - 2.0 / r)
    b = torch.minimum(b, bmax)
    total = torch.zeros_like(b)
    x, w = np.polynomial.legendre.leggauss(nodes)
    for xi, wi in zip(x, w):
        th = (xi + 1.0) * math.pi / 4.0
        u = math.sin(th) ** 2 / r
        inner = 1.0 - b * b * u * u * (1.0 - 2.0 * u)
        total += torch.where(inner > 0.0, wi * b * 2.0 / r * math.sin(th) * math.cos(th) / torch.sqrt(inner.clamp_min(1e-300)), 0.0)
    return total * math.pi / 4.0


class Lane:
    """Rays under way: tensors of one row a ray, kept to those still going."""

    def keep(self, mask):
        for k, v in vars(self).items():
            if isinstance(v, torch.Tensor):
                setattr(self, k, v[mask])


def begin(l, index, q):
    n = index.numel()
    l.index = index
    z = torch.zeros(n, device=index.device, dtype=F)
    l.color = torch.zeros(n, 3, device=index.device, dtype=F)
    l.through, l.limit = z + 1.0, z + q["cap"]
    return l


def schwarzschild(origin, direction, index, q, jump):
    """Launch from a static observer; with the jump, rays placed on the r = 30 sphere, those that miss it returned apart."""
    r0 = origin.norm(dim=1)
    l = begin(Lane(), index, q)
    l.e1 = origin / r0[:, None]
    dr = (direction * l.e1).sum(1)
    perp = direction - dr[:, None] * l.e1
    dphi = perp.norm(dim=1)
    l.e2 = perp / dphi.clamp_min(1e-12)[:, None]
    f0 = 1.0 - 2.0 / r0
    l.r, l.phi, l.vd, l.rd, l.pd = r0, torch.zeros_like(r0), (1.0 + dr) / f0.sqrt(), f0.sqrt() * dr, dphi / r0
    l.E, l.L = f0 * l.vd - l.rd, r0 * r0 * l.pd
    sky = (None, None)
    if jump:
        b = l.L.abs() / l.E
        turn = 29.0 / math.sqrt(1.0 - 2.0 / 29.0)
        out, miss = l.rd >= 0.0, b >= turn
        u = 1.0 / b.clamp_min(1.0)
        for _ in range(60):
            u = torch.where(miss, u - (1.0 - b * b * u * u * (1.0 - 2.0 * u)) / (-b * b * (2.0 * u - 6.0 * u * u)), u)
        here = sweep(r0, b)
        far = torch.where(out, here, 2.0 * (sweep(torch.where(miss, 1.0 / u, r0), b) - here) + here)
        lost = out | miss
        sky = index[lost], (torch.cos(far)[:, None] * l.e1 + torch.sin(far)[:, None] * l.e2)[lost]
        l.phi = sweep(torch.full_like(b, 30.0), b) - here
        l.r = torch.full_like(b, 30.0)
        f = 1.0 - 2.0 / 30.0
        l.rd = -torch.sqrt((l.E**2 - f * l.L**2 / 900.0).clamp_min(0.0))
        l.vd, l.pd = (l.E + l.rd) / f, l.L / 900.0
        l.keep(~lost)
    l.pos = polar(l)
    return l, sky


def polar(l):
    return l.r[:, None] * (torch.cos(l.phi)[:, None] * l.e1 + torch.sin(l.phi)[:, None] * l.e2)


def s_rate(y):
    r, _, vd, rd, pd = y
    vdd = -vd * vd / (r * r) + r * pd * pd
    return rd, pd, vdd, 2.0 * rd * vd / (r * r) + (1.0 - 2.0 / r) * vdd, -2.0 * rd * pd / r


def rk4(rate, y, h):
    k1 = rate(y)
    k2 = rate([a + 0.5 * h * b for a, b in zip(y, k1)])
    k3 = rate([a + 0.5 * h * b for a, b in zip(y, k2)])
    k4 = rate([a + h * b for a, b in zip(y, k3)])
    return [a + h / 6.0 * (p + 2.0 * q + 2.0 * r + s) for a, p, q, r, s in zip(y, k1, k2, k3, k4)]


def s_heading(l):
    c, s = torch.cos(l.phi)[:, None], torch.sin(l.phi)[:, None]
    radial, tangent = c * l.e1 + s * l.e2, c * l.e2 - s * l.e1
    return unit((l.rd / (1.0 - 2.0 / l.r).clamp_min(1e-6).sqrt())[:, None] * radial + (l.r * l.pd)[:, None] * tangent)


def s_advance(l, st, jump):
    coarse = (st["empty"] * l.r).clamp(0.02, st["empty_max"])
    fine = (f32(0.02) * l.r).clamp(f32(0.02), 0.5)
    h = torch.where(l.pos[:, 2].abs() > SLAB + coarse, coarse, fine)
    y = [l.r, l.phi, l.vd, l.rd, l.pd]
    z = rk4(s_rate, y, h)
    if jump:
        over = (z[0] >= HALF) & (z[3] > 0.0) & (l.r < HALF)
        z2 = rk4(s_rate, y, h * torch.where(over, (HALF - l.r) / (z[0] - l.r), 1.0))
        z = [torch.where(over, b, a) for a, b in zip(z, z2)]
    l.r, l.phi, l.vd, l.rd, l.pd = z
    return polar(l)


def kerr(origin, direction, index, q):
    """Launch from a static observer's tetrad in Boyer-Lindquist coordinates."""
    a = f32(q["spin"])
    l = begin(Lane(), index, q)
    rho2 = (origin * origin).sum(1)
    half = 0.5 * (rho2 - a * a)
    r = torch.sqrt(half + torch.sqrt(half * half + a * a * origin[:, 2] ** 2))
    th, ph = torch.acos((origin[:, 2] / rho2.sqrt()).clamp(-1.0, 1.0)), torch.atan2(origin[:, 1], origin[:, 0])
    rh, thh, phh = frame(th, ph)
    nr, nth, nph = ((direction * v).sum(1) for v in (rh, thh, phh))
    sg, dl, s2 = r * r + (a * torch.cos(th)) ** 2, r * r - 2.0 * r + a * a, torch.sin(th) ** 2
    gtt, gtp = -(1.0 - 2.0 * r / sg), -2.0 * a * r * s2 / sg
    gpp = (r * r + a * a + 2.0 * a * a * r * s2 / sg) * s2
    norm = torch.sqrt(gpp - gtp * gtp / gtt)
    pt, pp = 1.0 / torch.sqrt(-gtt) + nph * (-gtp / gtt) / norm, nph / norm
    l.E, l.L = -(gtt * pt + gtp * pp), gtp * pt + gpp * pp
    l.r, l.th, l.ph, l.pr, l.pt = r, th, ph, torch.sqrt(sg / dl) * nr, torch.sqrt(sg) * nth
    l.a = torch.full_like(r, a)
    l.horizon = 1.0 + torch.sqrt(1.0 - l.a**2)
    l.escape = torch.full_like(r, max(60.0, f32(q["distance"]) + 10.0) if "distance" in q else 60.0)
    l.pos = k_place(l)
    return l


def frame(th, ph):
    st, ct, sp, cp = torch.sin(th), torch.cos(th), torch.sin(ph), torch.cos(ph)
    return torch.stack([st * cp, st * sp, ct], 1), torch.stack([ct * cp, ct * sp, -st], 1), torch.stack([-sp, cp, 0.0 * sp], 1)


def k_place(l):
    w = torch.sqrt(l.r**2 + l.a**2) * torch.sin(l.th)
    return torch.stack([w * torch.cos(l.ph), w * torch.sin(l.ph), l.r * torch.cos(l.th)], 1)


def k_rate(l):
    a, E, L = l.a, l.E, l.L

    def rate(y):
        r, th, _, pr, pt = y
        st, ct = torch.sin(th), torch.cos(th)
        dl, sg, s2 = r * r - 2.0 * r + a * a, r * r + (a * ct) ** 2, (st * st).clamp_min(1e-12)
        p = (r * r + a * a) * E - a * L
        f = dl * pr * pr + pt * pt - p * p / dl + L * L / s2 - 2.0 * a * E * L + (a * E) ** 2 * s2
        dp = 2.0 * r - 2.0
        fr = dp * pr * pr - 4.0 * r * E * p / dl + p * p * dp / (dl * dl)
        fth = -2.0 * L * L * ct / (s2 * st.clamp_min(1e-9)) + 2.0 * (a * E) ** 2 * st * ct
        return (dl * pr / sg, pt / sg, (a * p / dl + L / s2 - a * E) / sg, (r * f / sg - 0.5 * fr) / sg,
                (-a * a * st * ct * f / sg - 0.5 * fth) / sg)

    return rate


def k_heading(l):
    rh, thh, phh = frame(l.th, l.ph)
    dr, dth, dph, _, _ = k_rate(l)((l.r, l.th, l.ph, l.pr, l.pt))
    return unit(dr[:, None] * rh + (l.r * dth)[:, None] * thh + (l.r * torch.sin(l.th) * dph)[:, None] * phh)


def k_advance(l):
    pole = (torch.sin(l.th) / 0.08).clamp(0.05, 1.0)
    h = (torch.minimum(f32(0.02) * l.r, 0.2 * (l.r - l.horizon)) * pole).clamp(0.002, 0.5)
    l.r, l.th, l.ph, l.pr, l.pt = rk4(k_rate(l), [l.r, l.th, l.ph, l.pr, l.pt], h)
    return k_place(l)


def texel(grid, n, p):
    """Trilinear interpolation between voxel centres, zero outside."""
    x = (p + HALF) / (2.0 * HALF) * n - 0.5
    b = x.floor()
    f, b = x - b, b.long()
    out = torch.zeros(p.shape[0], 4, device=p.device, dtype=F)
    for c in range(8):
        o = torch.tensor([c & 1, c >> 1 & 1, c >> 2], device=p.device)
        i = b + o
        w = torch.where(o.bool(), f, 1.0 - f).prod(1) * ((i >= 0) & (i < n)).all(1)
        i = i.clamp(0, n - 1)
        out += w[:, None] * grid[(i[:, 2] * n + i[:, 1]) * n + i[:, 0]].double()
    return out


def gather(l, which, lapse, heading, path, volume):
    e_grid, v_grid, n = volume
    p = l.pos[which]
    e, v = texel(e_grid, n, p), texel(v_grid, n, p)[:, :3]
    speed = v.norm(dim=1)
    ceiling = f32(0.85)
    beta = ceiling * torch.tanh(speed.clamp_max(8.0) / ceiling)
    scale = torch.where(speed > 0.0, beta / speed.clamp_min(1e-30), 0.0)
    gravity = lapse.clamp_min(0.0).sqrt()
    shift = gravity * torch.sqrt(1.0 - beta**2) / (1.0 + (heading * v).sum(1) * scale)
    bulk = (e[:, 3] / 40.0).clamp_max(1.0)
    g3 = gravity**3 + (shift**3 - gravity**3) * bulk
    has = e[:, 3] > 0.0
    k = torch.where(has, l.through[which] * g3 * path, 0.0)
    l.color[which] += e[:, :3] * k[:, None]
    l.through[which] *= torch.where(has, torch.exp(-f32(5e-4) * e[:, 3] * path), 1.0)


def blackbody():
    """Colour of a black body from 1000 to 40000 K, 256 entries log spaced, each rounded to half."""
    nm = np.arange(380.0, 781.0)

    def lobe(mu, s1, s2):
        return np.exp(-0.5 * ((nm - mu) / np.where(nm < mu, s1, s2)) ** 2)

    xyz = np.stack([1.056 * lobe(599.8, 37.9, 31.0) + 0.362 * lobe(442.0, 16.0, 26.7) - 0.065 * lobe(501.1, 20.4, 26.2),
                    0.821 * lobe(568.8, 46.9, 40.5) + 0.286 * lobe(530.9, 16.3, 31.1),
                    1.217 * lobe(437.0, 11.8, 36.0) + 0.681 * lobe(459.0, 26.0, 13.4)])
    t = np.exp(np.linspace(math.log(1000.0), math.log(40000.0), 256))[:, None]
    planck = 1.0 / ((nm * 1e-9) ** 5 * (np.exp(1.438776877e-2 / (nm * 1e-9 * t)) - 1.0))
    rgb = planck @ xyz.T @ np.array([[3.2406, -1.5372, -0.4986], [-0.9689, 1.8758, 0.0415], [0.0557, -0.2040, 1.0570]]).T
    rgb = rgb.clip(0.0)
    return (rgb / rgb.max(1, keepdims=True)).astype(np.float16).astype(np.float64)


def pcg4d(v):
    m = 0xFFFFFFFF
    x, y, z, w = ((c * 1664525 + 1013904223) & m for c in v)
    for shift in (True, False):
        x = (x + y * w) & m
        y = (y + z * x) & m
        z = (z + x * y) & m
        w = (w + y * z) & m
        if shift:
            x, y, z, w = (c ^ (c >> 16) for c in (x, y, z, w))
    return x, y, z, w


def unit_float(x):
    return (x >> 8).double() / 16777216.0


def stars(d, seed):
    a = d.abs()
    fx = (a[:, 0] >= a[:, 1]) & (a[:, 0] >= a[:, 2])
    axis = torch.where(fx, 0, torch.where(a[:, 1] >= a[:, 2], 1, 2))
    along = d.gather(1, axis[:, None])[:, 0]
    face = 2 * axis + (along <= 0.0)
    major = along.abs()
    sx = torch.where(axis == 0, d[:, 1], d[:, 0]) / major * 48.0 + 48.0
    sy = torch.where(axis == 2, d[:, 1], d[:, 2]) / major * 48.0 + 48.0
    cx, cy = sx.clamp_max(95.0).long(), sy.clamp_max(95.0).long()
    h = pcg4d((cx, cy, face, seed))
    dx, dy = sx - (cx + unit_float(h[1])), sy - (cy + unit_float(h[2]))
    bright = torch.where(h[0] <= 0x30000000, unit_float(h[3]) ** 3 * torch.exp(-40.0 * (dx * dx + dy * dy)), 0.0)
    c = torch.log(3000.0 + 9000.0 * unit_float(h[3] ^ h[1]))
    c = (c - math.log(1000.0)) / math.log(40.0) * 256.0 - 0.5
    table = torch.tensor(blackbody(), device=d.device)
    i = c.floor()
    lo, hi = table[i.long().clamp(0, 255)], table[(i.long() + 1).clamp(0, 255)]
    return (lo + (hi - lo) * (c - i)[:, None]) * bright[:, None]


def trace(l, spin, st, jump, volume, done):
    """Step every ray to its end; done(lane of the rays that ended, outcome 0 captured / 1 escaped / 2 out of steps, left the sphere)."""
    for step in range(st["cap"]):
        if l.index.numel() == 0:
            return
        before = l.pos
        l.pos = k_advance(l) if spin > 0.0 else s_advance(l, st, jump)
        path = (l.pos - before).norm(dim=1)
        captured = l.r <= (l.horizon + f32(0.05) if spin > 0.0 else CAPTURE)
        if volume is not None:
            p = l.pos.abs()
            which = ((p[:, 2] < SLAB) & (p[:, 0] < HALF) & (p[:, 1] < HALF) & (l.through > f32(0.004)) & ~captured).nonzero()[:, 0]
            if which.numel():
                sub = Lane()
                for k, v in vars(l).items():
                    setattr(sub, k, v[which])
                lapse = 1.0 - 2.0 * sub.r / (sub.r**2 + (sub.a * torch.cos(sub.th)) ** 2) if spin > 0.0 else 1.0 - 2.0 / sub.r
                gather(l, which, lapse, k_heading(sub) if spin > 0.0 else s_heading(sub), path[which], volume)
        sphere = (l.r >= HALF) & (l.rd > 0.0) if jump else torch.zeros_like(captured)
        escaped = ~captured & (sphere | (l.r >= (l.escape if spin > 0.0 else 60.0)))
        ended = captured | escaped | (step + 1 == st["cap"])
        if ended.any():
            out = Lane()
            for k, v in vars(l).items():
                setattr(out, k, v[ended])
            done(out, torch.where(captured, 0, torch.where(escaped, 1, 2))[ended], sphere[ended])
            l.keep(~ended)


def render(q, volume, device):
    """One served request in float64: (height * width, 4)."""
    origin, direction = camera_rays(q, device)
    n = origin.shape[0]
    image = torch.ones(n, 4, device=device, dtype=F)
    jump = q["spin"] == 0.0
    index = torch.arange(n, device=device)
    if jump:
        l, (lost, sky) = schwarzschild(origin, direction, index, q, True)
        image[lost, :3] = stars(sky, q["stars"]) * 1.5
    else:
        l = kerr(origin, direction, index, q)

    def done(o, outcome, sphere):
        if jump:
            b = o.L.abs() / o.E
            falls = (outcome == 0) | ((outcome == 2) & (o.rd < 0.0) & (b < f32(5.196152422706632)))
            phi = o.phi + sweep(torch.full_like(b, 30.0), b)
            sky = torch.cos(phi)[:, None] * o.e1 + torch.sin(phi)[:, None] * o.e2
            sky = torch.where(sphere[:, None], sky, s_heading(o))
        else:
            falls = (outcome == 0) | ((outcome == 2) & (o.pr < 0.0))
            sky = k_heading(o)
        light = stars(sky, q["stars"]) * (1.5 * o.through * ~falls)[:, None]
        image[o.index, :3] = o.color + light

    trace(l, q["spin"], settings(q["cap"]), jump, volume, done)
    return image


def exact(case, seed):
    device = device_of()
    if case["kind"] == "serve":
        q = requests(case, seed)
        # The float64 render takes about a second for each million rays.
        if sum(r["width"] * r["height"] for r in q) > 6_000_000 or len(q) > 8:
            return None
        volume = (*gas(128, seed, device), 128)
        return [render(r, volume, device) for r in q]
    if case["kind"] == "probes":
        launches = g.camera_grid(camera(seed), case["columns"], case["rows"], 16 / 9)
        o = torch.tensor(np.array([np.float32(l.origin) for l in launches], np.float64), device=device)
        d = unit(torch.tensor(np.array([np.float32(l.direction) for l in launches], np.float64), device=device))
        q = {"cap": 4096, "spin": case["spin"]}
        index = torch.arange(len(launches), device=device)
        l = kerr(o, d, index, q) if case["spin"] > 0.0 else schwarzschild(o, d, index, q, False)[0]
        out = {"position": torch.zeros_like(o), "direction": torch.zeros_like(o)}

        def done(e, outcome, sphere):
            out["position"][e.index] = e.pos
            out["direction"][e.index] = k_heading(e) if case["spin"] > 0.0 else s_heading(e)

        trace(l, case["spin"], settings(4096), False, None, done)
        return out
    if case["kind"] == "settle":
        return {"state": settle(particles(case["particles"], seed), case["dispatches"], seed, device), "respawns": None}
    return None  # sums and 8-bit pixels are whole numbers; a sequence's gas is a random deposit of them


def settle(records, dispatches, seed, device):
    """Dispatches of two substeps in float64: kick, drag, drift; captured, escaped or plunging particles start again."""
    s = torch.tensor(records, device=device).double()
    x, v = s[:, :3].clone(), s[:, 3:6].clone()
    event = torch.zeros(x.shape[0], device=device, dtype=torch.int64)
    dt, alpha = f32(0.1), f32(0.003)

    def shape(r):
        return (6.0 / r) ** 0.75 * (1.0 - torch.sqrt(6.0 / r)).clamp_min(f32(0.01)) ** 0.25

    scale = 8000.0 / shape(torch.tensor(6.0 * 49.0 / 36.0, dtype=F)).item()
    for _ in range(2 * dispatches):
        r = x.norm(dim=1)
        k = 1.0 / ((r - 2.0).clamp_min(1e-6) ** 2 * r)
        v = v - x * (k * dt)[:, None]
        v = v - v * (alpha * torch.sqrt(k) * dt)[:, None]
        step = v * dt
        tt = (step * step).sum(1).clamp_min(1e-12)
        along = (-(x * step).sum(1) / tt).clamp(0.0, 1.0)
        closest = (x + along[:, None] * step).norm(dim=1)
        x = x + step
        again = ((closest < CAPTURE) | (x.norm(dim=1) > 60.0) | (v.norm(dim=1) > 12.0)).nonzero()[:, 0]
        if again.numel():
            event[again] += 1
            lo, hi = seed & 0xFFFFFFFF, seed >> 32 & 0xFFFFFFFF
            h0 = pcg4d((again, event[again], torch.full_like(again, lo), torch.full_like(again, hi)))
            h1 = pcg4d((again, event[again], torch.full_like(again, lo ^ 0x9E3779B9), torch.full_like(again, hi)))
            u = [unit_float(c) for c in (*h0, *h1)]
            r = torch.sqrt(400.0 + 176.0 * u[0])
            phi = 2.0 * math.pi * u[1]
            a, b = torch.sqrt(-2.0 * torch.log(1.0 - u[2])), torch.sqrt(-2.0 * torch.log(1.0 - u[4]))
            g0, g1 = a * torch.cos(2.0 * math.pi * u[3]), a * torch.sin(2.0 * math.pi * u[3])
            g2, g3 = b * torch.cos(2.0 * math.pi * u[5]), b * torch.sin(2.0 * math.pi * u[5])
            vc = torch.sqrt(r) / (r - 2.0)
            sp = f32(0.02) * vc
            x[again] = torch.stack([r * torch.cos(phi), r * torch.sin(phi), f32(0.05) * r * g0], 1)
            v[again] = torch.stack([-vc * torch.sin(phi) + sp * g1, vc * torch.cos(phi) + sp * g2, sp * g3], 1)
    return torch.cat([x, v, (scale * shape(x.norm(dim=1)))[:, None]], 1)
