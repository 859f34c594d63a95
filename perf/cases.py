"""Workloads of the erosion library, through its public entry points.

Each case is one kind of work a program does with the library, at sizes from
the library's own workloads and tests:

  grid       a map eroded by some steps of hg_step (one layer), then read back
  batch      many terrains of uneven size stepped together
  layers     the reference's rock + dirt model with its default settings
  adjoint    one iteration of an inverse fit: forward, loss, backward
  particles  droplet erosion
  render     one ray-marched frame
  generate   the reference's terrain generator

A pass of a stepping case goes on from where the last one left its world, as
a program's main loop does, and reads the whole state back into device
buffers that the state keeps.

exact() gives the same outputs in 64 bits, from plain torch: the physics is
written out below from the shaders' formulas (one-layer and two-layer grid
step, its gradient through torch's autograd, the terrain generator).  The
droplets' per-texel order and the ray-marcher's bytes have no such value.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hydro-gen_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import hydrogen as H  # noqa: E402

FIELDS1 = ["rock", "water", "sediment", "flux_l", "flux_r", "flux_t", "flux_b", "vel_u", "vel_v"]
FIELDS2 = FIELDS1 + ["dirt", "sediment_dirt"]
CARRIED = FIELDS1[:7]
DEV = "cuda"


def f32(x):
    return float(np.float32(x))


# ---- the cases ------------------------------------------------------------------------

def listed():
    return [
        # an interactive tool's tick on a small map: launches and latency count
        dict(name="grid_256_tick", kind="grid", n=256, steps=8, physics="flow", mode="fused"),
        # plain virtual-pipe erosion of an ordinary map, no talus passes
        dict(name="grid_1024_flow", kind="grid", n=1024, steps=32, physics="flow", mode="fused"),
        # the headline workload: 4096^2, Bernoulli rain, talus slippage
        dict(name="grid_4096_storm", kind="grid", n=4096, steps=16, physics="storm", mode="fused"),
        # the large workload: 8192^2, uniform rain, talus slippage
        dict(name="grid_8192_talus", kind="grid", n=8192, steps=8, physics="talus", mode="fused"),
        # a map whose side the tiled kernels do not take: the per-pass kernels
        dict(name="grid_1000_passes", kind="grid", n=1000, steps=8, physics="storm", mode="plain"),
        # many terrains of uneven size and settings in one batch
        dict(name="batch_16_ragged", kind="batch", steps=16,
             sides="256,512,1024,2048,256,1024,512,2048,2048,512,256,1024,1024,2048,512,256"),
        # the reference's own model (rock and dirt, both talus layers, smoothing)
        dict(name="layers_2048", kind="layers", n=2048, steps=8, mode="fused"),
        # inverse erosion: per-cell solubility and initial heights, checkpoints
        dict(name="adjoint_1024_fit", kind="adjoint", n=1024, steps=32, ckpt=8, physics="flow"),
        # the same with talus slippage, the whole tape in memory
        dict(name="adjoint_2048_talus", kind="adjoint", n=2048, steps=12, ckpt=-1, physics="talus"),
        # droplet erosion at the reference's default count
        dict(name="particles_1024", kind="particles", n=1024, drops=262144, steps=8, warm=96),
        # one frame of the viewer
        dict(name="render_1080p", kind="render", n=1024, width=1920, height=1080),
        # "Generate map" of the reference's panel
        dict(name="generate_2048", kind="generate", n=2048, warp=1),
    ]


def _log_int(rng, lo, hi, mult):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(mult, int(round(v / mult)) * mult)


def draw(rng):
    kind = rng.choice(["grid", "grid", "passes", "batch", "layers", "adjoint", "particles", "render", "generate"])
    if kind in ("grid", "passes"):
        fused = kind == "grid"
        n = _log_int(rng, 128, 6000, 64) if fused else _log_int(rng, 72, 3000, 8)
        physics = rng.choice(["flow", "storm", "talus"])
        most = max(1, min(16 if physics == "storm" else 48, int(4.5e8 / (n * n))))
        return dict(kind="grid", n=n, steps=rng.randint(1, most), physics=physics,
                    mode="fused" if fused else "plain")
    if kind == "batch":
        sides = [rng.choice([256, 512, 1024, 2048, 64 * rng.randint(2, 20)]) for _ in range(rng.randint(2, 16))]
        return dict(kind="batch", steps=rng.randint(2, 16), sides=",".join(map(str, sides)))
    if kind == "layers":
        fused = rng.random() < 0.7
        n = _log_int(rng, 128, 2500, 64) if fused else _log_int(rng, 72, 1500, 8)
        return dict(kind="layers", n=n, steps=rng.randint(1, 12), mode="fused" if fused else "plain")
    if kind == "adjoint":
        steps = rng.randint(3, 24)
        return dict(kind="adjoint", n=_log_int(rng, 128, 1400, 64), steps=steps,
                    ckpt=rng.choice([-1, max(1, steps // 3), max(1, steps // 2)]),
                    physics=rng.choice(["flow", "talus"]))
    if kind == "particles":
        return dict(kind="particles", n=_log_int(rng, 192, 1600, 8), drops=_log_int(rng, 4096, 262144, 1),
                    steps=rng.randint(1, 12), warm=32)
    if kind == "render":
        return dict(kind="render", n=_log_int(rng, 256, 2048, 8), width=rng.randint(320, 1920),
                    height=rng.randint(200, 1080))
    return dict(kind="generate", n=_log_int(rng, 128, 4096, 8), warp=rng.choice([1, 1, 2]))


# ---- inputs ---------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _fractal(n, g, octaves=6, wavelength=128):
    """Octaves of smooth noise (gain 1/2), scaled to [0, 1]: the statistics of
    the workloads' fBm heightmaps."""
    out = torch.zeros(n, n, device=DEV)
    amp = 1.0
    for o in range(octaves):
        cell = max(2, wavelength >> o)
        m = n // cell + 4
        grid = torch.randn(1, 1, m, m, generator=g, device=DEV)
        up = torch.nn.functional.interpolate(grid, scale_factor=cell, mode="bicubic", align_corners=False)
        out += amp * up[0, 0, cell:cell + n, cell:cell + n]
        amp *= 0.5
    lo, hi = out.min(), out.max()
    return (out - lo) / (hi - lo)


def _ground(n, seed):
    """Rock in [0, 64] under a flood, deeper in the lowest third: it runs off
    into the valleys over the passes and leaves films and puddles behind."""
    g = _gen(seed)
    rock = (64.0 * _fractal(n, g)).contiguous()
    level = 0.3 * 64.0
    water = 1.0 + 0.25 * torch.clamp(level - rock, min=0.0)
    return rock, water.contiguous()


def _physics(name):
    """Parameters of the grid workloads, as floats of the settings struct."""
    p = dict(Kc=0.1, Ks=0.05, Kd=0.05, Ke=0.015, G=9.81, dt=0.02, EK=1.0, alpha=math.atan(0.65), slip=0.0,
             rain="uniform", amount=0.01, prob=0.0)
    if name in ("storm", "talus"):
        p["slip"] = 0.3
    if name == "storm":
        p.update(rain="bernoulli", amount=0.5, prob=0.001)
    return p


def _terrain_physics(i, seed):
    """The ragged batch's per-terrain settings."""
    rng = random.Random(seed * 1009 + i)
    lu = lambda a, b: math.exp(rng.uniform(math.log(a), math.log(b)))  # noqa: E731
    p = _physics("storm")
    p.update(Kc=lu(0.05, 0.5), Ks=lu(0.01, 0.1), Kd=lu(0.01, 0.1), Ke=rng.uniform(0.005, 0.03),
             alpha=math.atan(rng.uniform(0.4, 0.9)))
    return p


def _apply(w, p, seed, terrain_id=0):
    s = H.settings_config1()
    s.Kc, s.Ke, s.G, s.d_t, s.ENERGY_KEPT = p["Kc"], p["Ke"], p["G"], p["dt"], p["EK"]
    s.Ks[0] = s.Ks[1] = p["Ks"]
    s.Kd[0] = s.Kd[1] = p["Kd"]
    s.Kalpha[0] = s.Kalpha[1] = p["alpha"]
    s.Kspeed[0] = p["slip"]
    w.set_erosion(s)
    w.set_rain(H.rain_uniform(p["amount"], 1))
    mode = H.RAIN_UNIFORM if p["rain"] == "uniform" else H.RAIN_BERNOULLI
    w.set_options(H.options(mode, p=p["prob"], seed=seed, terrain_id=terrain_id))


def _load(w, fields):
    torch.cuda.synchronize()  # the inputs were made on torch's stream
    for name, t in fields.items():
        w.upload_device(name, t.data_ptr())
    w.sync()


def _layer_settings():
    s = H.ErosionSettings()
    H.check(H.lib.hg_default_erosion_settings(ctypes.byref(s)))
    return s


def _layer_ground(n, seed):
    """Rock in [0, 160], up to 2 of dirt, water as in _ground."""
    g = _gen(seed)
    rock = (160.0 * _fractal(n, g, wavelength=256)).contiguous()
    dirt = (2.0 * _fractal(n, g, octaves=4, wavelength=64)).contiguous()
    water = 0.25 + 0.25 * torch.clamp(48.0 - rock, min=0.0)
    return rock, dirt, water.contiguous()


def _sides(case):
    return [int(x) for x in case["sides"].split(",")]


def _mode(case):
    return H.MODE_FUSED if case["mode"] == "fused" else H.MODE_PLAIN


def _map(case, seed):
    return H.map_settings(hmap_dims=(case["n"], case["n"]), seed=(seed % 997) / 100.0, domain_warp=case["warp"])


def _fit_inputs(case, seed):
    n = case["n"]
    rock, water = _ground(n, seed)
    g = _gen(seed + 77)
    ks = (0.05 * torch.exp(_fractal(n, g, octaves=3, wavelength=256) - 0.5)).contiguous()
    target = (rock + 0.2 * (_fractal(n, g, octaves=4) - 0.5)).contiguous()
    return rock, water, ks, target


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "kind": kind}
    if kind == "grid":
        n = case["n"]
        w = H.World(n)
        _apply(w, _physics(case["physics"]), seed)
        rock, water = _ground(n, seed)
        _load(w, {"rock": rock, "water": water})
        st.update(w=w, out=torch.empty(len(FIELDS1), n, n, device=DEV))
    elif kind == "batch":
        worlds, outs = [], []
        for i, n in enumerate(_sides(case)):
            w = H.World(n)
            _apply(w, _terrain_physics(i, seed), seed, terrain_id=i)
            rock, water = _ground(n, seed + 31 * i)
            _load(w, {"rock": rock, "water": water})
            worlds.append(w)
            outs.append(torch.empty(len(FIELDS1), n, n, device=DEV))
        st.update(worlds=worlds, batch=H.Batch(worlds), outs=outs)
    elif kind == "layers":
        n = case["n"]
        w = H.World(n, layers=2)
        w.set_erosion(_layer_settings())
        w.set_rain(H.rain_uniform(0.01, 1))
        w.set_options(H.options(H.RAIN_UNIFORM))
        rock, dirt, water = _layer_ground(n, seed)
        _load(w, {"rock": rock, "dirt": dirt, "water": water})
        st.update(w=w, out=torch.empty(len(FIELDS2), n, n, device=DEV))
    elif kind == "adjoint":
        n = case["n"]
        w = H.World(n)
        _apply(w, _physics(case["physics"]), seed)
        rock, water, ks, target = _fit_inputs(case, seed)
        _load(w, {"rock": rock, "water": water, "ks": ks})
        tape = H.Tape(w, case["steps"], case["ckpt"])
        st.update(w=w, tape=tape, rock0=rock, water0=water, zero=torch.zeros(n, n, device=DEV), target=target,
                  g=torch.empty(n, n, device=DEV), out=torch.empty(len(FIELDS1) + 2, n, n, device=DEV))
        torch.cuda.synchronize()
    elif kind == "particles":
        n = case["n"]
        w = H.World(n, layers=2)
        rock, dirt, _ = _layer_ground(n, seed)
        _load(w, {"rock": rock, "dirt": dirt})
        w.particles_init(case["drops"])
        w.set_erosion(H.settings_particles())
        w.set_options(H.options(H.RAIN_UNIFORM, seed=seed))
        w.step(case["warm"], H.MODE_PARTICLES)  # droplets spread out, some gathered in the valleys
        w.sync()
        st.update(w=w, out=torch.empty(5, n, n, device=DEV))
    elif kind == "render":
        n, wd, ht = case["n"], case["width"], case["height"]
        w = H.World(n, layers=2)
        rock, dirt, _ = _layer_ground(n, seed)
        water = torch.clamp(60.0 - (rock + dirt), min=0.0).contiguous()
        _load(w, {"rock": rock, "dirt": dirt, "water": water})
        k = n / 1024.0
        cam = H.camera((150.0 * k, 170.0, 150.0 * k), (1.0, -0.35, 1.0), aspect=wd / ht)
        st.update(w=w, cam=cam, out=torch.empty(ht, wd, 4, dtype=torch.uint8, device=DEV))
    elif kind == "generate":
        n = case["n"]
        st.update(w=H.World(n, layers=2), map=_map(case, seed), out=torch.empty(2, n, n, device=DEV))
    else:
        raise ValueError(kind)
    return st


# ---- one pass ---------------------------------------------------------------------------

def _read(w, names, out):
    for i, name in enumerate(names):
        w.download_device(name, out[i].data_ptr())
    return {name: out[i] for i, name in enumerate(names)}


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "grid":
        st["w"].step(case["steps"], _mode(case))
        return _read(st["w"], FIELDS1, st["out"])
    if kind == "batch":
        st["batch"].step(case["steps"])
        for w, o in zip(st["worlds"], st["outs"]):
            _read(w, FIELDS1, o)
        return list(st["outs"])
    if kind == "layers":
        st["w"].step(case["steps"], _mode(case))
        return _read(st["w"], FIELDS2, st["out"])
    if kind == "adjoint":
        w, out = st["w"], st["out"]
        w.upload_device("rock", st["rock0"].data_ptr())
        w.upload_device("water", st["water0"].data_ptr())
        for f in CARRIED[2:]:
            w.upload_device(f, st["zero"].data_ptr())
        w.step_count = 0
        st["tape"].forward()
        loss = H.mse(w, st["target"].data_ptr(), st["g"].data_ptr())
        st["tape"].backward(st["g"].data_ptr(), out[-2].data_ptr(), out[-1].data_ptr())
        return dict(_read(w, FIELDS1, out), loss=loss, dks=out[-2], drock0=out[-1])
    if kind == "particles":
        st["w"].step(case["steps"], H.MODE_PARTICLES)
        return _read(st["w"], ["rock", "dirt", "water", "momentum_x", "momentum_y"], st["out"])
    if kind == "render":
        H.check(H.lib.hg_render_device(st["w"].h, ctypes.byref(st["cam"]), case["width"], case["height"],
                                       ctypes.c_void_p(st["out"].data_ptr()), None))
        return st["out"]
    st["w"].init_reference_heightmap(st["map"])
    return _read(st["w"], ["rock", "dirt"], st["out"])


def work(case):
    """Bytes: the state read and written once per step (9 fields, 11 with the
    dirt layer), the result written once; a reversed step reads a state and
    the step's intermediates and reads and writes an adjoint state.  Flops:
    the arithmetic of the passes per cell, droplet or pixel."""
    kind = case["kind"]
    if kind == "batch":
        cells = sum(n * n for n in _sides(case))
        return {"bytes": cells * (72.0 * case["steps"] + 36), "flops": cells * case["steps"] * 320.0}
    cells = float(case["n"]) ** 2
    if kind == "grid":
        fl = 180.0 if case["physics"] == "flow" else 320.0
        return {"bytes": cells * (72.0 * case["steps"] + 36), "flops": cells * case["steps"] * fl}
    if kind == "layers":
        return {"bytes": cells * (88.0 * case["steps"] + 44), "flops": cells * case["steps"] * 550.0}
    if kind == "adjoint":
        return {"bytes": cells * (case["steps"] * (72.0 + 100.0) + 44), "flops": cells * case["steps"] * 1000.0}
    if kind == "particles":
        d = float(case["drops"])
        return {"bytes": case["steps"] * (d * (80 + 96) + cells * 56) + cells * 20,
                "flops": case["steps"] * (d * 600.0 + cells * 350.0)}
    if kind == "render":
        px = float(case["width"]) * case["height"]
        return {"bytes": cells * 12 + px * 4, "flops": px * 6000.0}
    return {"bytes": cells * 8, "flops": cells * 8 * 110.0 * (4 if case["warp"] == 1 else 6)}


# ---- 64-bit values ------------------------------------------------------------------------

FAR = f32(999999999999.0)
D8 = [(-1, 0), (1, 0), (0, 1), (0, -1), (-1, 1), (1, 1), (-1, -1), (1, -1)]  # L R T B LT RT LB RB; +y is up


def _nb(a, dx, dy, fill):
    """The value at (x + dx, y + dy), `fill` outside the grid."""
    p = torch.nn.functional.pad(a[None, None], (1, 1, 1, 1), value=fill)[0, 0]
    n0, n1 = a.shape
    return p[1 + dy:1 + dy + n0, 1 + dx:1 + dx + n1]


def _pos(x):
    return torch.where(x > 0, x, torch.zeros_like(x))


def _sqrt(x):
    """sqrt with derivative 0 at 0."""
    ok = x > 0
    return torch.where(ok, torch.sqrt(torch.where(ok, x, torch.ones_like(x))), torch.zeros_like(x))


def _philox_words(n, step, terrain, seed):
    """Philox4x32-10 words of every cell: counter (x / 4, y, step, terrain), key (seed); cell x takes word x % 4."""
    M = 0xFFFFFFFF

    def mulhilo(m, a):
        al, ah = a & 0xFFFF, a >> 16
        t = m * al
        return (m * ah + (t >> 16)) >> 16, (m * a) & M

    y, x = torch.meshgrid(torch.arange(n, device=DEV), torch.arange(n // 4, device=DEV), indexing="ij")
    c = [x, y, torch.full_like(x, step & M), torch.full_like(x, terrain)]
    k0, k1 = seed & M, (seed >> 32) & M
    for _ in range(10):
        h0, l0 = mulhilo(0xD2511F53, c[0])
        h1, l1 = mulhilo(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return torch.stack(c, dim=-1).reshape(n, n)


def _rain(p, n, step, seed, terrain):
    if p["rain"] == "uniform":
        return f32(p["amount"])
    thr = math.floor(f32(p["prob"]) * 4294967296.0)
    return torch.where(_philox_words(n, step, terrain, seed) < thr, f32(p["amount"]), 0.0).double()


def _talus(terr, drops, dt, alpha, slip):
    """Outflows toward the eight neighbours of the layer of height `terr`."""
    hmax = torch.zeros_like(terr)
    for d in drops:
        hmax = torch.maximum(hmax, d)
    H_ = torch.minimum(terr, hmax)
    sharp, bk, marks = torch.ones_like(terr), torch.zeros_like(terr), []
    for k, d in enumerate(drops):
        down = d > 0
        slope = torch.where(down, d, torch.zeros_like(d)) / (1.0 if k < 4 else math.sqrt(2.0))
        a = torch.atan(slope)
        m = down & (a > alpha)
        sharp = torch.where(m, torch.maximum(sharp, 1.0 + a - alpha), sharp)
        bk = bk + torch.where(m, d, torch.zeros_like(d))
        marks.append(m)
    S = dt * slip * sharp ** 3 * H_ / 2.0
    safe = torch.where(bk > 0, bk, torch.ones_like(bk))
    return [torch.where(m, S * d / safe, torch.zeros_like(d)) for m, d in zip(marks, drops)]


def _move(h, out):
    opposite = [1, 0, 3, 2, 7, 6, 5, 4]
    total = h
    for k, (dx, dy) in enumerate(D8):
        total = total - out[k] + _nb(out[opposite[k]], dx, dy, 0.0)
    return total


def _step64(s, p, rain, ks=None):
    """One step of the grid model; `s`: dict of fields, with dirt in the two-layer model."""
    two = "dirt" in s
    n = s["rock"].shape[0]
    dt, G, EK = f32(p["dt"]), f32(p["G"]), f32(p["EK"])
    d1 = s["water"] + rain
    ground = s["rock"] + s["dirt"] if two else s["rock"]
    total = ground + d1
    old = [s["flux_l"], s["flux_r"], s["flux_t"], s["flux_b"]]
    g = [_pos(EK * old[k] + dt * G * (total - _nb(total, *D8[k], FAR))) for k in range(4)]
    inflow = [_nb(old[(1, 0, 3, 2)[k]], *D8[k], 0.0) for k in range(4)]
    sum_in = inflow[0] + inflow[1] + inflow[2] + inflow[3]
    sum_out = g[0] + g[1] + g[2] + g[3]
    den = sum_out * dt
    short = d1 < den
    K = torch.where(short, d1 / torch.where(short, den, torch.ones_like(den)), torch.ones_like(den))
    d2 = _pos(d1 + dt * (sum_in - sum_out * K))
    vz = d1 + d2
    wet = vz > 0
    vs = torch.where(wet, vz, torch.ones_like(vz))
    u = torch.where(wet, (inflow[0] - old[0] + old[1] - inflow[1]) / vs, torch.zeros_like(vz))
    v = torch.where(wet, (inflow[3] - old[3] + old[2] - inflow[2]) / vs, torch.zeros_like(vz))
    flux = [a * K for a in g]
    # erosion
    speed = _sqrt(u * u + v * v)
    t = torch.clamp((torch.clamp(vz, min=f32(5e-4)) - f32(1e-3)) / (f32(5e-4) - f32(1e-3)), 0.0, 1.0)
    speed = torch.where(vz < f32(1e-3), speed * (1.0 - t * t * (3.0 - 2.0 * t)), speed)
    dx = _nb(ground, 1, 0, 0.0) - _nb(ground, -1, 0, 0.0)
    dz = _nb(ground, 0, 1, 0.0) - _nb(ground, 0, -1, 0.0)
    cos2 = 16.0 / (4.0 * dx * dx + 16.0 + 4.0 * dz * dz)
    tilt = _sqrt(1.0 - cos2)
    tilt = torch.where(tilt > f32(0.02), tilt, torch.full_like(tilt, f32(0.02)))
    cap = _pos(f32(p["Kc"]) * tilt * speed)
    new = {"water": d2 * (1.0 - f32(p["Ke"]) * dt)}
    kls = dt * (ks if ks is not None else f32(p["Ks"]))
    if two:
        gone, cont, h, sed = torch.zeros_like(cap), torch.ones_like(cap, dtype=torch.bool), {}, {}
        for name, sn, kl, kd in (("dirt", "sediment_dirt", dt * f32(p["Ks1"]), dt * f32(p["Kd1"])),
                                 ("rock", "sediment", kls, dt * f32(p["Kd"]))):
            c = _pos(cap - gone)
            more = c > s[sn]
            take = kl * (c - s[sn])
            short_ = more & (s[name] - take < 0)
            h1 = torch.where(more, torch.where(short_, torch.zeros_like(c), s[name] - take),
                             s[name] + kd * (s[sn] - c))
            s1 = torch.where(more, torch.where(short_, s[sn] + s[name], s[sn] + take), s[sn] - kd * (s[sn] - c))
            h[name] = torch.where(cont, h1, s[name])
            sed[sn] = torch.where(cont, s1, s[sn])
            gone = torch.where(cont & short_, gone + s[name], gone)
            cont = cont & ~(more & ~short_)
        conv = sed["sediment"] * f32(p["Kconv"]) * dt
        rock, dirt = h["rock"], h["dirt"]
        seds = {"sediment": sed["sediment"] - conv, "sediment_dirt": sed["sediment_dirt"] + conv}
    else:
        more = cap > s["sediment"]
        take = kls * (cap - s["sediment"])
        give = dt * f32(p["Kd"]) * (s["sediment"] - cap)
        short_ = more & (s["rock"] - take < 0)
        rock = torch.where(more, torch.where(short_, torch.zeros_like(cap), s["rock"] - take), s["rock"] + give)
        seds = {"sediment": torch.where(more, torch.where(short_, s["sediment"] + s["rock"], s["sediment"] + take),
                                        s["sediment"] - give)}
        dirt = None
    # semi-Lagrangian sediment transport
    ar = torch.arange(n, device=DEV, dtype=torch.float64)
    px = torch.clamp(ar[None, :] - u * dt, 0.0, n - 1.0)
    py = torch.clamp(ar[:, None] - v * dt, 0.0, n - 1.0)
    ix, iy = px.detach().floor().long(), py.detach().floor().long()
    fx, fy = px - ix, py - iy
    ix1, iy1 = torch.clamp(ix + 1, max=n - 1), torch.clamp(iy + 1, max=n - 1)  # weight 0 where clamped
    for name, f in seds.items():
        flat = f.reshape(-1)
        a = flat[iy * n + ix] * (1 - fx) + flat[iy * n + ix1] * fx
        b = flat[iy1 * n + ix] * (1 - fx) + flat[iy1 * n + ix1] * fx
        new[name] = a * (1 - fy) + b * fy
    # talus passes and smoothing
    if p["slip"] != 0.0:
        rock = _move(rock, _talus(rock, [rock - _nb(rock, *d, FAR) for d in D8], dt, f32(p["alpha"]), f32(p["slip"])))
    if two:
        drops = [(rock - _nb(rock, *d, FAR)) + (dirt - _nb(dirt, *d, FAR)) for d in D8]
        dirt = _move(dirt, _talus(dirt, drops, dt, f32(p["alpha1"]), f32(p["slip1"])))
        m = min(max(f32(p["slip1"]) * dt, 0.0), 1.0)
        dr = [rock - _nb(rock, *d, 0.0) for d in D8[:4]]
        dd = [(dirt - _nb(dirt, *d, 0.0)) + a for d, a in zip(D8[:4], dr)]
        inner = torch.zeros_like(rock, dtype=torch.bool)
        inner[1:-1, 1:-1] = True
        sm = []
        for h, d in ((rock, dr), (dirt, dd)):
            mean = torch.abs((d[0] + d[1] + d[2] + d[3]) / 4.0)
            peak = (((-d[0] > mean) | (-d[1] > mean)) & (d[0] * d[1] > 0)) | \
                   (((-d[2] > mean) | (-d[3] > mean)) & (d[2] * d[3] > 0))
            avg = (h + _nb(h, -1, 0, 0.0) + _nb(h, 1, 0, 0.0) + _nb(h, 0, 1, 0.0) + _nb(h, 0, -1, 0.0)) / 5.0
            sm.append(torch.where(inner & peak, m * avg + (1.0 - m) * h, h))
        rock, dirt = sm
        new["dirt"] = dirt
    new.update(rock=rock, flux_l=flux[0], flux_r=flux[1], flux_t=flux[2], flux_b=flux[3], vel_u=u, vel_v=v)
    return new


def _start64(fields, names):
    ref = next(iter(fields.values()))
    return {k: fields[k].double() if k in fields else torch.zeros_like(ref, dtype=torch.float64) for k in names}


def _grid64(rock, water, p, steps, seed, terrain=0):
    s = _start64({"rock": rock, "water": water}, FIELDS1)
    for k in range(steps):
        s = _step64(s, p, _rain(p, rock.shape[0], k + 1, seed, terrain))
    return s


def _layer_params():
    s = _layer_settings()
    return dict(Kc=s.Kc, Ks=s.Ks[0], Kd=s.Kd[0], Ks1=s.Ks[1], Kd1=s.Kd[1], Ke=s.Ke, G=s.G, dt=s.d_t,
                EK=s.ENERGY_KEPT, Kconv=s.Kconv, alpha=s.Kalpha[0], slip=s.Kspeed[0], alpha1=s.Kalpha[1],
                slip1=s.Kspeed[1])


def _adjoint64(case, seed):
    rock, water, ks, target = _fit_inputs(case, seed)
    p, n = _physics(case["physics"]), case["n"]
    ks = ks.double().requires_grad_(True)
    r0 = rock.double().requires_grad_(True)
    s = _start64({"rock": rock, "water": water}, FIELDS1)
    s["rock"] = r0
    for k in range(case["steps"]):
        s = torch.utils.checkpoint.checkpoint(_step64, s, p, _rain(p, n, k + 1, seed, 0), ks, use_reentrant=False)
    e = s["rock"] - target.double()
    loss = (e * e).mean()
    gks, gr = torch.autograd.grad(loss, [ks, r0])
    return dict({k: t.detach() for k, t in s.items()}, loss=float(loss.detach()), dks=gks, drock0=gr)


def _elias(ix, iy):
    M = 0xFFFFFFFF
    out = []
    for a, b in ((3, 311), (37, 113)):
        v = (ix * a + iy * b) & M
        v = ((v << 13) & M) ^ v
        t = ((v * v) & M) * 15731 + 789221
        v = (v * (t & M) + 1376312589) & 0x0FFFFFFF
        out.append(-1.0 + 2.0 * v.double() / 268435455.0)
    return out


def _gnoise64(px, py):
    ix, iy = px.floor(), py.floor()
    fx, fy = px - ix, py - iy
    ix, iy = ix.long(), iy.long()
    ux = fx ** 3 * (fx * (fx * 6 - 15) + 10)
    uy = fy ** 3 * (fy * (fy * 6 - 15) + 10)
    dux = 30 * fx * fx * (fx * (fx - 2) + 1)
    duy = 30 * fy * fy * (fy * (fy - 2) + 1)
    a, b, c, e = _elias(ix, iy), _elias(ix + 1, iy), _elias(ix, iy + 1), _elias(ix + 1, iy + 1)
    va = a[0] * fx + a[1] * fy
    vb = b[0] * (fx - 1) + b[1] * fy
    vc = c[0] * fx + c[1] * (fy - 1)
    vd = e[0] * (fx - 1) + e[1] * (fy - 1)
    k, uu = va - vb - vc + vd, ux * uy
    val = va + ux * (vb - va) + uy * (vc - va) + uu * k
    ddx = a[0] + ux * (b[0] - a[0]) + uy * (c[0] - a[0]) + uu * (a[0] - b[0] - c[0] + e[0]) + dux * (uy * k + vb - va)
    ddy = a[1] + ux * (b[1] - a[1]) + uy * (c[1] - a[1]) + uu * (a[1] - b[1] - c[1] + e[1]) + duy * (ux * k + vc - va)
    return val, ddx, ddy


def _fbm64(x, y, m, eroded):
    off = f32(f32(m.seed) * 100.0)
    x, y = x + off, y + off
    acc, amp, norm, sx, sy = 0.0, 1.0, 1.0, 0.0, 0.0
    freq = 1.5 if eroded else 1.0
    for _ in range(m.octaves):
        v, dx, dy = _gnoise64(x * freq * m.scale, y * freq * m.scale)
        t = (v + 1) / 2 * amp
        if eroded:
            sx, sy = sx + dx, sy + dy
            t = t / (1 + (sx * sx + sy * sy))
        acc = acc + t
        freq *= m.lacunarity
        amp *= m.persistance
        norm += amp
    return acc / norm


def _generate64(case, seed):
    m, n = _map(case, seed), case["n"]
    y, x = torch.meshgrid(torch.arange(n, device=DEV, dtype=torch.float64),
                          torch.arange(n, device=DEV, dtype=torch.float64), indexing="ij")
    ws = m.domain_warp_scale
    wx, wy = _fbm64(x + 2.3, y + 2.9, m, False), _fbm64(x - 3.1, y - 4.3, m, False)
    if m.domain_warp == 2:
        wx, wy = (_fbm64(x + ws * wx - 5.7, y + ws * wy + 27.9, m, False),
                  _fbm64(x + ws * wx + 11.5, y + ws * wy - 23.7, m, False))
    val = _fbm64(x + ws * wx, y + ws * wy, m, True)
    val = val * (torch.exp(val) - 1) / 1.718  # mask_exp
    val = val * ((((val + 0.5) ** 3 - 0.125) / 3.25) * 0.55 + 0.45)  # mask_power
    hm = m.height_mult + 2.0 + 1.25 + 2.0
    rock = torch.clamp(val * m.max_height * hm, max=m.max_height)
    return {"rock": rock, "dirt": (_fbm64(x + 13.7, y + 27.1, m, False) + 1.5) * m.max_dirt}


def exact(case, seed):
    kind = case["kind"]
    if kind == "adjoint":
        return _adjoint64(case, seed)
    with torch.no_grad():
        if kind == "grid":
            rock, water = _ground(case["n"], seed)
            return _grid64(rock, water, _physics(case["physics"]), case["steps"], seed)
        if kind == "batch":
            out = []
            for i, n in enumerate(_sides(case)):
                rock, water = _ground(n, seed + 31 * i)
                s = _grid64(rock, water, _terrain_physics(i, seed), case["steps"], seed, terrain=i)
                out.append(torch.stack([s[f] for f in FIELDS1]))
            return out
        if kind == "layers":
            rock, dirt, water = _layer_ground(case["n"], seed)
            s, p = _start64({"rock": rock, "dirt": dirt, "water": water}, FIELDS2), _layer_params()
            for _ in range(case["steps"]):
                s = _step64(s, p, f32(0.01))
            return s
        if kind == "generate":
            return _generate64(case, seed)
    return None
