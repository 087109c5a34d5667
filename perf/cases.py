"""The work that users of the solvers have them do, as cases that can be timed and checked.

A case is a dict of plain values; ``prepare`` makes what a program has in hand before the call
(a session with its model, receivers, display buffers), ``run`` is one pass through the public
entry points, ``exact`` is the same pass in 64-bit torch arithmetic, written here from the
scheme's equations.  Kinds of cases:

* ``shot3d``  - a stretch of a 3-D shot: gather opened, steps run, traces fetched;
* ``live3d``  - the interactive 3-D loop: one step, then the receiver spread is sampled;
* ``batch3d`` - windows of a survey stepped together;
* ``views3d`` - one displayed frame: view extraction, slice shading, raymarched volume;
* ``upload3d`` - a new earth model handed to a session as three host volumes;
* ``shot2d``  - a stretch of a 2-D shot, in the three schemes, one or several sources;
* ``live2d``  - the interactive 2-D loop: one step, the wavefield texture, the receivers.

A solver session carries its state from call to call, so every pass of the stepping kinds goes
on where the last one stopped.  Sessions start from seeded smooth wavefields in a seeded model
rather than from silence, so that every cell, the absorbing layers and the surfaces carry
waves from the first step on.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cmakepro_cuda_seissim_v2_b200 import capi, capi2d, seis2d, seis3d

W = (1225.0 / 1024.0, -245.0 / 3072.0, 49.0 / 5120.0, -5.0 / 7168.0)
FIELDS_2D = ("vx_1", "vx_2", "vz_1", "vz_2", "sxx_1", "sxx_2", "szz_1", "szz_2", "sxz_1", "sxz_2")
TOTALS_2D = ("vx", "vz", "sigmaxx", "sigmazz", "sigmaxz")
L2_BYTES = 126_000_000


# ---- the cases ----------------------------------------------------------------------------

def listed():
    return [
        # The largest grid the solver takes (36 M nodes), all six faces absorbing: the long
        # production shot, bound by memory and by the passes' arithmetic.
        {"name": "shot3d_size_cap", "kind": "shot3d", "nx": 300, "ny": 300, "nz": 400, "pml": 20, "surface": False,
         "walls": False, "storage": "fp32", "source": "explosion", "steps": 20, "rx": 20, "ry": 15, "stride": 1},
        # The grid that a new workspace opens with, with a 20-cell layer and a free surface, replayed for a
        # progress interval of 64 steps and recorded every second step.
        {"name": "shot3d_default", "kind": "shot3d", "nx": 300, "ny": 50, "nz": 300, "pml": 20, "surface": True,
         "walls": False, "storage": "fp32", "source": "explosion", "steps": 64, "rx": 50, "ry": 3, "stride": 2},
        # One window of a windowed survey with odd sides, in the 16-bit memory mode.
        {"name": "shot3d_window_bf16", "kind": "shot3d", "nx": 213, "ny": 199, "nz": 187, "pml": 20, "surface": True,
         "walls": False, "storage": "bf16_cpml", "source": "explosion", "steps": 16, "rx": 50, "ry": 3, "stride": 2},
        # A small exploratory model: everything is latency and launches.
        {"name": "shot3d_small", "kind": "shot3d", "nx": 40, "ny": 32, "nz": 36, "pml": 8, "surface": True,
         "walls": False, "storage": "fp32", "source": "force", "steps": 64, "rx": 5, "ry": 3, "stride": 1},
        # Slip walls instead of absorbing layers, odd sides, fewer steps than one graph replay.
        {"name": "shot3d_walls", "kind": "shot3d", "nx": 97, "ny": 61, "nz": 83, "pml": 8, "surface": False,
         "walls": True, "storage": "fp32", "source": "force", "steps": 40, "rx": 20, "ry": 3, "stride": 1},
        # The interactive loop on the workspace's default context: one step, then a receiver sample.
        {"name": "live3d", "kind": "live3d", "nx": 300, "ny": 50, "nz": 300, "pml": 12, "surface": True,
         "walls": False, "storage": "fp32", "source": "explosion", "rx": 50, "ry": 3},
        # Three uneven windows of a survey on one device.
        {"name": "batch3d_windows", "kind": "batch3d", "windows": "161x120x171,205x97x160,180x133x187", "pml": 20,
         "surface": True, "storage": "fp32", "source": "explosion", "steps": 12, "rx": 50, "ry": 3, "stride": 2},
        # One displayed frame of the default workspace: slices and a 640 x 640 volume.
        {"name": "views3d", "kind": "views3d", "nx": 300, "ny": 50, "nz": 300, "pml": 12, "surface": True,
         "component": 0, "material": 5, "width": 640, "height": 640},
        # A new window's model, from host volumes.
        {"name": "upload3d", "kind": "upload3d", "nx": 245, "ny": 133, "nz": 187, "pml": 20, "surface": True},
        # The 2-D free-surface shot with its receiver line.
        {"name": "shot2d_two_layer", "kind": "shot2d", "nx": 440, "nz": 420, "npml": 20, "flag": 3, "up": True,
         "type": capi2d.EXPLOSIVE, "steps": 256, "receivers": 200, "stride": 1, "sources": 0},
        # A large 2-D section in the hybrid scheme, beyond what the L2 cache holds.
        {"name": "shot2d_large_hybrid", "kind": "shot2d", "nx": 1601, "nz": 1203, "npml": 30, "flag": 2, "up": False,
         "type": capi2d.VERTICAL_FORCE, "steps": 48, "receivers": 160, "stride": 2, "sources": 0},
        # The interactive 2-D loop on a small grid.
        {"name": "live2d", "kind": "live2d", "nx": 120, "nz": 100, "npml": 12, "flag": 1, "up": False,
         "type": capi2d.ROTATED_FORCE, "receivers": 40},
    ]


def draw(rng):
    """One more case of the same ranges."""

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["shot3d"] * 4 + ["shot2d"] * 4 + ["live3d", "live2d", "batch3d", "views3d", "upload3d"])
    if kind in ("shot2d", "live2d"):
        flag = rng.choice([1, 2, 3])
        up = flag == 3 and rng.random() < 0.8
        npml = rng.randint(8, 30)
        small = kind == "live2d"
        c = {"kind": kind, "nx": size(90, 700 if small else 2000), "nz": size(90, 700 if small else 1500),
             "npml": npml, "flag": flag, "up": up, "type": rng.randint(0, 4), "receivers": rng.randint(1, 200)}
        if not small:
            cells = c["nx"] * c["nz"]
            c["sources"] = rng.choice([0, 0, 0, 6])
            c["steps"] = max(2, min(size(20, 400), 100_000_000 // cells))
            c["stride"] = rng.choice([1, 2, 3])
        return c
    surface = rng.random() < 0.6
    if kind == "batch3d":
        sizes = [(size(30, 200), size(24, 160), size(30, 190)) for _ in range(rng.randint(2, 5))]
        pml = rng.randint(8, 24)
        cells = sum((x + 2 * pml) * (y + 2 * pml) * (z + 2 * pml) for x, y, z in sizes)
        return {"kind": kind, "windows": ",".join("%dx%dx%d" % s for s in sizes), "pml": pml, "surface": surface,
                "storage": rng.choice(["fp32", "fp32", "bf16_cpml"]), "source": rng.choice(["explosion", "force"]),
                "steps": max(2, min(rng.randint(4, 80), 700_000_000 // cells)), "rx": rng.randint(2, 50), "ry": rng.randint(1, 3), "stride": rng.choice([1, 2])}
    c = {"kind": kind, "nx": size(20, 300), "ny": size(20, 300), "nz": size(20, 300), "pml": rng.randint(8, 30),
         "surface": surface}
    if kind == "upload3d":
        return c
    if kind == "views3d":
        c.update(component=rng.randint(0, 4), material=rng.randint(5, 7), width=size(160, 1536), height=size(160, 1536))
        return c
    walls = rng.random() < 0.2
    c.update(walls=walls, surface=surface and not walls, storage=rng.choice(["fp32", "fp32", "bf16_cpml"]),
             source=rng.choice(["explosion", "force"]), rx=rng.randint(1, 50), ry=rng.randint(1, 6))
    if kind == "shot3d":
        cells = (c["nx"] + 2 * c["pml"]) * (c["ny"] + 2 * c["pml"]) * (c["nz"] + 2 * c["pml"])
        c["steps"] = max(2, min(size(8, 160), 700_000_000 // cells))
        c["stride"] = rng.choice([1, 2])
    return c


# ---- inputs -------------------------------------------------------------------------------

def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1009 + salt)
    return g


def _smooth(shape, cells, g):
    """Smooth noise in [-1, 1]: uniform draws every `cells` cells, interpolated linearly."""
    coarse = [max(2, -(-n // cells) + 1) for n in shape]
    x = torch.rand([1, 1] + coarse, generator=g, device="cuda") * 2 - 1
    mode = "trilinear" if len(shape) == 3 else "bilinear"
    return torch.nn.functional.interpolate(x, size=tuple(shape), mode=mode, align_corners=True)[0, 0].contiguous()


def _taper(shape, cells=6):
    """1 inside, falling to 0 towards the edges of the array (float32)."""
    out = torch.ones((), device="cuda")
    for a, n in enumerate(shape):
        d = torch.arange(n, device="cuda", dtype=torch.float32)
        d = torch.clamp(torch.minimum(d, n - 1 - d) / cells, max=1.0)
        w = torch.sin(0.5 * math.pi * d) ** 2
        out = out * w.reshape([-1 if b == a else 1 for b in range(len(shape))])
    return out


class _DeviceArray:
    """A solver buffer as torch sees it (no copy); the tensors made from it keep its owner alive."""

    def __init__(self, owner, address, shape, strides):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "strides": tuple(strides), "typestr": "<f4",
                                         "data": (int(address), False), "version": 3}


def _device(owner, address, shape, strides):
    return torch.as_tensor(_DeviceArray(owner, address, shape, strides), device="cuda")


def _case3d(c):
    """The full set of a 3-D case's values."""
    full = {"walls": False, "storage": "fp32", "source": "explosion", "rx": 50, "ry": 3, "steps": 1, "stride": 1}
    full.update(c)
    return full


def _windows(c):
    for k, text in enumerate(c["windows"].split(",")):
        nx, ny, nz = (int(v) for v in text.split("x"))
        yield k, _case3d({**c, "nx": nx, "ny": ny, "nz": nz})


def _model3d(c, seed):
    """vp, vs, rho [nz][ny][nx] float32 on the device: a depth gradient with smooth variations."""
    g = _generator(seed, 1)
    shape = (c["nz"], c["ny"], c["nx"])
    depth = torch.linspace(1800.0, 4200.0, c["nz"], device="cuda").reshape(-1, 1, 1)
    vp = (depth * (1 + 0.08 * _smooth(shape, 8, g))).contiguous()
    vs = vp * (0.55 + 0.04 * _smooth(shape, 12, g))
    rho = 310.0 * torch.sqrt(torch.sqrt(vp))
    return vp, vs.contiguous(), rho.contiguous()


def _context3d(c, vp_max):
    ctx = seis3d.default_context(nx3D=c["nx"], ny3D=c["ny"], nz3D=c["nz"], spacing3D=10.0, pml3D=c["pml"],
                                 freeSurface3D=int(c["surface"]), reflecting3D=int(c["walls"]),
                                 modelKind3D=capi.MODEL_IMPORTED, maxVp3D=vp_max, frequency3D=15.0)
    return seis3d.validate_context3D(ctx)


def _source3d(c):
    kind = {"explosion": capi.SOURCE_EXPLOSION, "force": capi.SOURCE_FORCE}[c["source"]]
    return {"x": c["nx"] // 2, "y": c["ny"] // 2 - 1, "z": max(2, c["nz"] // 3), "kind": kind,
            "amplitude": 1.0e8 if c["source"] == "explosion" else 1.0e4, "direction": (0.3, -0.5, 0.8)}


def _receivers3d(c):
    """A surface spread of rx x ry receivers over the physical model."""
    xs = np.unique(np.linspace(1, c["nx"] - 2, c["rx"]).astype(int))
    ys = np.unique(np.linspace(1, c["ny"] - 2, c["ry"]).astype(int))
    return np.array([(x, y, 0) for y in ys for x in xs], dtype=np.int32)


def _first_step(dt, frequency, steps):
    """The steps of a first pass straddle the source's peak."""
    return max(0, int(1.2 / frequency / dt) - steps // 2)


def _initial3d(c, seed, g_shape):
    """Nine seeded wavefields [gz][gy][gx] float32, zero in the four ghost cells of every side."""
    g = _generator(seed, 2)
    inner = [n - 8 for n in g_shape]
    taper = _taper(inner)
    out = []
    for k in range(9):
        f = torch.zeros(g_shape, device="cuda")
        f[4:-4, 4:-4, 4:-4] = _smooth(inner, 9, g) * taper * (1e-3 if k < 3 else 6e3)
        out.append(f)
    return out


def _session3d(c, seed):
    vp, vs, rho = _model3d(c, seed)
    ctx = _context3d(c, float(vp.max()))
    storage = {"fp32": capi.STORAGE_FP32, "bf16_cpml": capi.STORAGE_BF16_CPML}[c["storage"]]
    s = seis3d.Session(ctx, storage=storage)
    s.upload_volumes(vp.cpu().numpy(), vs.cpu().numpy(), rho.cpu().numpy())
    s.set_receivers(_receivers3d(c))
    v = s.views()
    x = s.context
    shape, strides = (x.gz3D, x.gy3D, x.gx3D), (4 * v.plane, 4 * v.pitch, 4)
    fields = {name: _device(s, v.field3D[k], shape, strides) for k, name in enumerate(capi.FIELDS)}
    for f, values in zip(fields.values(), _initial3d(c, seed, shape)):
        f.copy_(values)
    torch.cuda.synchronize()
    q = _source3d(c)
    src = seis3d.default_source(x3D=q["x"], y3D=q["y"], z3D=q["z"], kind3D=q["kind"], amplitude3D=q["amplitude"],
                                direction3D=q["direction"])
    materials = [_device(s, p, shape, strides) for p in (v.inverseDensity3D, v.lambda3D, v.mu3D)]
    return {"session": s, "source": src, "fields": fields, "materials": materials,
            "step": _first_step(x.dt3D, 15.0, c["steps"]), "steps": c["steps"], "stride": c["stride"]}


def _arrays2d(c, seed):
    """The host arrays of a 2-D context (float32), flat [z * NX + x] volumes and damping lines."""
    nx, nz, npml = c["nx"], c["nz"], c["npml"]
    g = _generator(seed, 3)
    depth = torch.linspace(2000.0, 3800.0, nz, device="cuda").reshape(-1, 1)
    vp = (depth * (1 + 0.06 * _smooth((nz, nx), 10, g))).cpu().numpy()
    vs = vp * np.float32(0.57)
    rho = (np.float32(310.0) * np.sqrt(np.sqrt(vp))).astype(np.float32)
    mu, l2m = rho * vs * vs, rho * vp * vp
    lam = l2m - np.float32(2.0) * mu
    h, dt, f0, nt = 5.0, 0.0005, 20.0, 2000
    lines = {n: np.zeros(k, np.float32) for n, k in (("dx", nx), ("dx_half", nx), ("dz", nz), ("dz_half", nz))}
    d_max = 3.0 * float(vp.max()) * 16.12 * 3.5 / (2.0 * npml * h)
    for i in range(npml):
        whole, half = d_max * ((npml - i) / npml) ** 2.5, d_max * ((npml - i - 0.5) / npml) ** 2.5
        for n, v in (("dx", whole), ("dz", whole), ("dx_half", half), ("dz_half", half)):
            lines[n][i] = lines[n][-1 - i] = v
    row = l2m[npml].astype(np.float64), lam[npml].astype(np.float64)
    t = np.arange(nt) * dt - 1.0 / f0
    a = (math.pi * f0 * t) ** 2
    fs = npml if c["flag"] == 3 and c["up"] else 0
    sx, sz = nx // 2 + 1, min(nz - 12, fs + 12 + nz // 8)
    rcv = np.unique(np.linspace(5, nx - 6, c["receivers"]).astype(int)) + (fs + 6) * nx
    w = [np.float32(np.float32(v) / np.float32(h)) for v in W]
    return {"rho": rho.ravel(), "mu": mu.ravel(), "lambda_": lam.ravel(), "lambda2mu": l2m.ravel(), **lines,
            "dp_flat": ((row[0] ** 2 - row[1] ** 2) / row[0]).astype(np.float32), "h": h, "dt": float(np.float32(dt)),
            "nt": nt, "f0": f0, "wavelet": ((1 - 2 * a) * np.exp(-a)).astype(np.float32), "weights": w,
            "src": (sx, sz), "rcv": rcv.astype(np.int32)}


def _sources2d(c, a):
    """(flat index, time, peak frequency, amplitude) of the simultaneous sources of a case."""
    sx, sz = a["src"]
    return [((sz + k % 3) * c["nx"] + max(6, min(c["nx"] - 7, sx + 7 * (k - 3))), 0.03 + 0.002 * k, 20.0 + k, 1.0 + 0.1 * k)
            for k in range(c.get("sources", 0))]


def _initial2d(c, seed):
    """Seeded wavefields of a 2-D case: the ten split halves, silent above a free surface."""
    g = _generator(seed, 4)
    shape = (c["nz"], c["nx"])
    taper = torch.zeros(shape, device="cuda")
    top = c["npml"] if c["flag"] == 3 and c["up"] else 4
    taper[top:-4, 4:-4] = _taper((c["nz"] - 4 - top, c["nx"] - 8))
    return {n: _smooth(shape, 9, g) * taper * (0.5 if n[0] == "v" else 3e6) for n in FIELDS_2D}


def _session2d(c, seed):
    a = _arrays2d(c, seed)
    ctx = seis2d.SimulationContext(NX=c["nx"], NZ=c["nz"], total_grid=c["nx"] * c["nz"], h=a["h"], dt=a["dt"],
                                   nt=a["nt"], npml=c["npml"], flag_type=c["flag"], upFlag=c["up"])
    for n in ("rho", "mu", "lambda_", "lambda2mu", "dp_flat", "dx", "dx_half", "dz", "dz_half", "wavelet"):
        setattr(ctx, n, a[n])
    ctx.c1_h, ctx.c2_h, ctx.c3_h, ctx.c4_h = (float(w) for w in a["weights"])
    ctx.src_z_idx = a["src"][1]
    ctx.src_idx = a["src"][1] * c["nx"] + a["src"][0]
    ctx.src_type, ctx.src_angle = c["type"], 30.0
    ctx.rcv_grid_idx = a["rcv"]
    ctx.num_rcv = int(a["rcv"].size)
    gpu = seis2d.GPUSimData()
    seis2d.initializeGpuSimulation(gpu, ctx)
    v = gpu.views()
    names = FIELDS_2D + (TOTALS_2D if c["flag"] == 2 else ())
    fields = {n: _device(gpu, v.field[capi2d.FIELD[n]], (c["nz"], c["nx"]), (4 * c["nx"], 4)) for n in names}
    first = _initial2d(c, seed)
    for n in FIELDS_2D:
        fields[n].copy_(first[n])
    if c["flag"] == 2:
        for k, n in enumerate(TOTALS_2D):
            fields[n].copy_(first[FIELDS_2D[2 * k]] + first[FIELDS_2D[2 * k + 1]])
    sources = _sources2d(c, a)
    if sources:
        seis2d.setActiveSources(gpu, sources)
    torch.cuda.synchronize()
    return {"gpu": gpu, "context": ctx, "fields": fields, "step": _first_step(a["dt"], 1.2 * a["f0"], c.get("steps", 1)),
            "steps": c.get("steps", 1), "stride": c.get("stride", 1), "active": len(sources) or -1,
            "receivers": ctx.num_rcv}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("shot2d", "live2d"):
        state = _session2d(case, seed)
        if kind == "live2d":
            state["texture"] = torch.zeros((case["nz"], case["nx"], 4), dtype=torch.uint8, device="cuda")
    elif kind == "batch3d":
        shots = [_session3d(c, seed * 16 + k) for k, c in _windows(case)]
        state = {"shots": shots, "batch": seis3d.Batch([s["session"] for s in shots]), "step": shots[0]["step"]}
    elif kind == "upload3d":
        c = _case3d(case)
        vp, vs, rho = _model3d(c, seed)
        s = seis3d.Session(_context3d(c, float(vp.max())))
        v, x = s.views(), s.context
        shape, strides = (x.gz3D, x.gy3D, x.gx3D), (4 * v.plane, 4 * v.pitch, 4)
        state = {"session": s, "model": [a.cpu().numpy() for a in (vp, vs, rho)],
                 "materials": [_device(s, p, shape, strides) for p in (v.inverseDensity3D, v.lambda3D, v.mu3D)]}
    else:
        c = _case3d(case)
        state = _session3d(c, seed)
        if kind == "views3d":
            s = state["session"]
            layout = seis3d.make_view_layout3D(s.context)
            state.update(layout=layout, slices=(c["nx"] // 2, c["ny"] // 2, c["nz"] // 3), component=c["component"],
                         material=c["material"], width=c["width"], height=c["height"],
                         views=torch.zeros((layout.totalSamples3D, 2), device="cuda"),
                         slice_pixels=torch.zeros((layout.volumeOffset3D, 4), dtype=torch.uint8, device="cuda"),
                         volume_pixels=torch.zeros((c["height"], c["width"], 4), dtype=torch.uint8, device="cuda"))
    state["kind"] = kind
    torch.cuda.synchronize()
    return state


# ---- one pass -----------------------------------------------------------------------------

def run(state):
    return {"shot3d": _run_shot3d, "live3d": _run_live3d, "batch3d": _run_batch3d, "views3d": _run_views3d,
            "upload3d": _run_upload3d, "shot2d": _run_shot2d, "live2d": _run_live2d}[state["kind"]](state)


def _run_shot3d(state):
    s, n = state["session"], state["steps"]
    s.gather_begin(state["stride"], max(1, n // state["stride"]))
    s.run_steps(state["source"], state["step"], n)
    state["step"] += n
    return {"gather": s.gather_fetch(), **state["fields"]}


def _run_live3d(state):
    s = state["session"]
    s.run_step(state["source"], state["step"])
    state["step"] += 1
    return {"samples": s.sample_receivers(), **state["fields"]}


def _run_batch3d(state):
    shots, n, stride = state["shots"], state["shots"][0]["steps"], state["shots"][0]["stride"]
    for shot in shots:
        shot["session"].gather_begin(stride, max(1, n // stride))
    state["batch"].run_steps([shot["source"] for shot in shots], state["step"], n)
    state["step"] += n
    state["batch"].synchronize()
    return [{"gather": shot["session"].gather_fetch(), **shot["fields"]} for shot in shots]


def _run_views3d(state):
    s, layout = state["session"], state["layout"]
    stats = s.extract_views(state["views"].data_ptr(), layout, state["slices"], state["component"], state["material"], True)
    display = seis3d.default_display(component3D=state["component"], scale3D=stats["maximum"],
                                     materialRange3D=list(stats["material_range"]),
                                     volumeRequestedWidth3D=state["width"], volumeRequestedHeight3D=state["height"])
    t, u, w, h = seis3d.make_display_uniforms(s.context, layout, display)
    s.shade_slices(layout, state["views"].data_ptr(), t, u.scale3D, u.gain3D, capi.PIXELS_RGBA8,
                   state["slice_pixels"].data_ptr())
    s.render_volume(layout, state["views"].data_ptr(), t, u, w, h, capi.PIXELS_RGBA8, state["volume_pixels"].data_ptr())
    s.synchronize()
    return {"wave": state["views"][:, 0], "material": state["views"][:, 1], "slices": state["slice_pixels"],
            "volume": state["volume_pixels"], "maximum": stats["maximum"],
            "velocity_maximum": stats["velocity_maximum"], "range": stats["material_range"]}


def _run_upload3d(state):
    state["session"].upload_volumes(*state["model"])
    return dict(zip(("inverse_density", "lambda", "mu"), state["materials"]))


def _run_shot2d(state):
    gpu, n, stride = state["gpu"], state["steps"], state["stride"]
    samples = -(-n // stride)
    seis2d.gatherBegin(gpu, state["step"], stride, samples)
    seis2d.runGpuSimulationSteps(gpu, state["step"], n, state["context"], state["active"])
    state["step"] += n
    vx, vz, taken = seis2d.gatherFetch(gpu, samples)
    return {"trace_vx": vx, "trace_vz": vz, "taken": taken, **state["fields"]}


def _run_live2d(state):
    gpu = state["gpu"]
    seis2d.runGpuSimulationStep(gpu, state["step"], state["context"], state["active"])
    state["step"] += 1
    seis2d.generateWavefieldTextureOnGpu(gpu, state["texture"].data_ptr(), 0.5, 0)
    vx, vz = seis2d.recordReceiverStepOnGpu(gpu, state["receivers"])
    return {"receivers_vx": vx, "receivers_vz": vz, "texture": state["texture"], **state["fields"]}


# ---- what a pass cannot do without -------------------------------------------------------

def _work_step3d(c):
    """(bytes of the state, bytes of one step, operations of one step): nine fields read and
    written, three materials read, six memories per layer cell read and written."""
    p = 0 if c["walls"] else c["pml"]
    ax, ay, az = c["nx"] + 2 * p, c["ny"] + 2 * p, c["nz"] + (1 if c["surface"] else 2) * p
    cells = ax * ay * az
    slab = 2 * p * ay * az + 2 * p * ax * az + (1 if c["surface"] else 2) * p * ax * ay
    memory = 2 if c["storage"] == "bf16_cpml" else 4
    traffic = 84 * cells + 12 * memory * slab
    return 48 * cells + 6 * memory * slab, traffic, 18 * 16 * cells + 60 * cells + 24 * slab


def work(case):
    kind = case["kind"]
    if kind in ("shot2d", "live2d"):
        cells, steps = case["nx"] * case["nz"], case.get("steps", 1)
        totals = 5 if case["flag"] == 2 else 0
        state = 4 * cells * (14 + totals)
        once = 4 * cells * (24 + 2 * totals)     # fields read and written, materials read
        # A state that the L2 cache holds has to be read and written once a pass, a larger one every step.
        per_step = 4 * cells * ((24 if case["flag"] != 2 else 15) if state > L2_BYTES else 0)
        extra = 4 * cells if kind == "live2d" else 0
        return {"bytes": max(once, per_step * steps) + extra, "flops": steps * cells * (8 * 16 + 40)}
    if kind == "batch3d":
        parts = [_work_step3d(c) for _, c in _windows(case)]
        return {"bytes": sum(p[1] for p in parts) * case["steps"], "flops": sum(p[2] for p in parts) * case["steps"]}
    c = _case3d(case)
    if kind == "upload3d":
        p = c["pml"]
        padded = (c["nx"] + 2 * p + 8) * (c["ny"] + 2 * p + 8) * (c["nz"] + (1 if c["surface"] else 2) * p + 8)
        return {"bytes": 12 * c["nx"] * c["ny"] * c["nz"] + 12 * padded, "flops": 8 * c["nx"] * c["ny"] * c["nz"]}
    state, step, flops = _work_step3d(c)
    if kind == "views3d":
        p = c["pml"]
        nx, ny, nz = c["nx"] + 2 * p, c["ny"] + 2 * p, c["nz"] + (1 if c["surface"] else 2) * p
        samples = min(256, nx) * min(256, ny) * min(256, nz) + nx * nz + ny * nz + nx * ny
        # Velocities and materials read, samples written, read by the shaders, pixels written.
        return {"bytes": 24 * nx * ny * nz + 16 * samples + 4 * (nx * nz + ny * nz + nx * ny) + 4 * c["width"] * c["height"],
                "flops": 8 * 20 * samples + 192 * 60 * c["width"] * c["height"]}
    steps = c["steps"]
    bytes_ = step * steps if state > L2_BYTES else 84 * state / 48
    return {"bytes": bytes_, "flops": flops * steps}


# ---- the same in 64 bits -------------------------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind in ("shot2d", "live2d"):
        return _exact2d(case, seed)
    if kind == "batch3d":
        c0 = next(_windows(case))[1]
        first = None
        out = []
        for k, c in _windows(case):
            m = _Scheme3d(c, seed * 16 + k)
            if first is None:
                first = _first_step(m.dt, 15.0, c0["steps"])
            out.append(m.shot(first))
        return out
    c = _case3d(case)
    if kind == "upload3d":
        m = _Scheme3d(c, seed, fields=False)
        return {"inverse_density": m.b, "lambda": m.lam, "mu": m.mu}
    m = _Scheme3d(c, seed)
    if kind == "views3d":
        return m.views()
    first = _first_step(m.dt, 15.0, c["steps"])
    if kind == "live3d":
        m.steps(first, 1)
        return {"samples": m.sample(), **m.named()}
    return m.shot(first)


class _Scheme3d:
    """The 3-D velocity-stress scheme in float64 on the padded grid."""

    def __init__(self, c, seed, fields=True):
        self.c = c
        vp, vs, rho = _model3d(c, seed)
        vp_max = float(vp.max())
        p = self.p = 0 if c["walls"] else c["pml"]
        self.ox = self.oy = p + 4
        self.oz = 4 if c["surface"] else p + 4
        self.n = (c["nz"] + (1 if c["surface"] else 2) * p + 8, c["ny"] + 2 * p + 8, c["nx"] + 2 * p + 8)
        weights = sum(abs(w) for w in W)
        safe = float(np.float32(0.85)) * 10.0 / (math.sqrt(3.0) * vp_max * weights)
        self.dt = float(np.float32(math.floor(safe * 1e6) * 1e-6))
        self.frequency, self.h, self.vp_max = 15.0, 10.0, vp_max
        r64, p64, s64 = rho.double(), vp.double(), vs.double()
        b, lam, mu = 1 / r64, r64 * (p64 * p64 - 2 * s64 * s64), r64 * s64 * s64
        at = [torch.clamp(torch.arange(n, device="cuda") - o, 0, k - 1)
              for n, o, k in zip(self.n, (self.oz, self.oy, self.ox), vp.shape)]
        # Materials of the padding are those of the nearest physical cell.
        self.b, self.lam, self.mu = (m[at[0]][:, at[1]][:, :, at[2]] for m in (b, lam, mu))
        if fields:
            self.f = [x.double() for x in _initial3d(c, seed, self.n)]

    def named(self):
        return dict(zip(capi.FIELDS, self.f))

    # axis: 0 = x, 1 = y, 2 = z; arrays are [z][y][x].
    def _shift(self, f, axis, k):
        start = [4, 4, 4]
        start[2 - axis] += k
        return f[tuple(slice(s, s + n - 8) for s, n in zip(start, self.n))]

    def _d(self, f, axis, forward):
        at = 1 if forward else 0
        out = W[0] * (self._shift(f, axis, at) - self._shift(f, axis, at - 1))
        for r in range(1, 4):
            out += W[r] * (self._shift(f, axis, at + r) - self._shift(f, axis, at - 1 - r))
        return out / self.h

    def _profiles(self):
        """a, b, 1/kappa of every axis at whole (0) and half (1) nodes of the interior."""
        out = []
        for axis in range(3):
            n = self.n[2 - axis]
            sigma_max = -4.0 * self.vp_max * math.log(1e-6) / (2.0 * self.p * self.h)
            pair = []
            for half in (0, 1):
                x = torch.arange(n, device="cuda", dtype=torch.float64) + 0.5 * half
                d = (x - (n - 4 - self.p - 0.5)) / self.p
                if not (axis == 2 and self.c["surface"]):
                    d = torch.maximum(d, (4 + self.p - 0.5 - x) / self.p)
                d = torch.clamp(d, 0, 1)
                sigma, kappa = sigma_max * d ** 3, 1 + 2 * d ** 3
                alpha = torch.where(d > 0, math.pi * self.frequency * (1 - d), torch.zeros_like(d))
                b = torch.exp(-(sigma / kappa + alpha) * self.dt)
                a = torch.where(sigma > 0, sigma * (b - 1) / (kappa * (sigma + kappa * alpha)).clamp(min=1e-300),
                                torch.zeros_like(d))
                shape = [1, 1, 1]
                shape[2 - axis] = n - 8
                pair.append([v[4:-4].reshape(shape) for v in (a, b, 1 / kappa)])
            out.append(pair)
        return out

    def _setup(self):
        I = self._shift  # noqa: E741
        b = I(self.b, 0, 0)
        self.c_face = [2 * b * q / (b + q) for q in (I(self.b, a, 1) for a in range(3))]
        r = 1 / self.mu

        def edge(p, q):
            corner = [4, 4, 4]
            corner[2 - p] += 1
            corner[2 - q] += 1
            both = r[tuple(slice(s, s + n - 8) for s, n in zip(corner, self.n))]
            return 4 / (I(r, 0, 0) + I(r, p, 1) + I(r, q, 1) + both)

        self.mu_xy, self.mu_yz, self.mu_xz = edge(0, 1), edge(1, 2), edge(0, 2)
        self.psi = {}
        self.profiles = self._profiles() if self.p else None

    def _layer(self, key, d, axis, half):
        if not self.p:
            return d
        a, b, ik = self.profiles[axis][half]
        m = self.psi.get(key)
        m = a * d if m is None else m.mul_(b).add_(a * d)
        self.psi[key] = m
        return ik * d + m

    def _source(self, time):
        """{(dz, dy, dx): value} of the 27 nodes."""
        q = _source3d(self.c)
        phase = math.pi * self.frequency * (time - 1.2 / self.frequency)
        ricker = (1 - 2 * phase * phase) * math.exp(-phase * phase)
        norm = (1 + 2 * math.exp(-0.5)) ** 3
        near = range(-1, 2)
        return {(dz, dy, dx): self.dt * q["amplitude"] * ricker * math.exp(-0.5 * (dx * dx + dy * dy + dz * dz)) / norm
                for dz in near for dy in near for dx in near}

    def _stress_surface(self):
        f = self.f
        s = (slice(4, -4), slice(4, -4))
        f[5][4][s] = 0
        for k in range(1, 5):
            for i in (3, 4, 6):
                f[i][4 - k][s] = f[i][4 + k][s]
            f[5][4 - k][s] = -f[5][4 + k][s]
            for i in (7, 8):
                f[i][4 - k][s] = -f[i][3 + k][s]

    def _velocity_surface(self):
        vx, vy, vz = self.f[:3]
        s = (slice(4, -4), slice(4, -4))

        def d(f, plane, axis, forward):
            at = 1 if forward else 0
            n = [self.n[1] - 8, self.n[2] - 8]

            def w(k):
                o = [4, 4]
                o[1 - axis] += k
                return f[plane, o[0]:o[0] + n[0], o[1]:o[1] + n[1]]

            return sum(W[r] * (w(at + r) - w(at - 1 - r)) for r in range(4)) / self.h

        ex, ey = d(vx, 4, 0, False), d(vy, 4, 1, False)
        dz_vx = -(1.5 * d(vz, 4, 0, True) - 0.5 * d(vz, 5, 0, True))
        dz_vy = -(1.5 * d(vz, 4, 1, True) - 0.5 * d(vz, 5, 1, True))
        lam, mu = self.lam[4][s], self.mu[4][s]
        dz_vz = -lam / (lam + 2 * mu) * (ex + ey)
        for k in range(1, 5):
            vx[4 - k][s] = vx[4 + k][s] - 2 * k * self.h * dz_vx
            vy[4 - k][s] = vy[4 + k][s] - 2 * k * self.h * dz_vy
            vz[4 - k][s] = vz[3 + k][s] - (2 * k - 1) * self.h * dz_vz

    def _walls(self, fields):
        for axis in range(3):
            n = self.n[2 - axis]
            high = n - 5
            for i in fields:
                f = self.f[i].movedim(2 - axis, 0)
                half = i == axis if i < 3 else {6: axis != 2, 7: axis != 0, 8: axis != 1}.get(i, False)
                sign = -1.0 if half else 1.0
                for d in range(1, 5):
                    f[4 - d] = 0 if half and d == 1 else sign * f[4 + d - 1 - int(half)]
                for d in range(1, 5):
                    f[high + d] = sign * f[high + 1 - d - int(half)]
                if half:
                    f[high] = 0

    def _images(self, velocities):
        if self.c["surface"]:
            self._velocity_surface() if velocities else self._stress_surface()
        if self.c["walls"]:
            self._walls(range(3) if velocities else range(3, 9))

    def steps(self, first, count, after=None):
        self._setup()
        q = _source3d(self.c)
        sx, sy, sz = q["x"] + self.ox, q["y"] + self.oy, q["z"] + self.oz
        f, inner, dt = self.f, (slice(4, -4),) * 3, self.dt
        vx, vy, vz, sxx, syy, szz, sxy, syz, sxz = f
        top = self.c["surface"]
        lam, mu = self.lam[inner], self.mu[inner]
        for step in range(first, first + count):
            self._images(False)
            terms = ((vx, ((sxx, True), (sxy, False), (sxz, False))), (vy, ((sxy, False), (syy, True), (syz, False))),
                     (vz, ((sxz, False), (syz, False), (szz, True))))
            new = []
            for v, (field, parts) in enumerate(terms):
                total = 0
                for axis, (s, forward) in enumerate(parts):
                    total = total + self._layer((v, axis), self._d(s, axis, forward), axis, int(v == axis))
                new.append((field, total))
            for v, (field, total) in enumerate(new):
                field[inner] += dt * self.c_face[v] * total
            if self.c["source"] == "force":
                for (dz, dy, dx), value in self._source(step * dt).items():
                    z, y, x = sz + dz, sy + dy, sx + dx
                    if all(4 <= i < n - 4 for i, n in zip((z, y, x), self.n)):
                        for v in range(3):
                            f[v][z, y, x] += value * q["direction"][v] * self.c_face[v][z - 4, y - 4, x - 4]
            self._images(True)
            d = [[self._layer((3 + v, a), self._d(f[v], a, a != v), a, int(a != v)) for a in range(3)] for v in range(3)]
            if top:
                k = (0,)
                d[2][2][k] = -lam[k] / (lam[k] + 2 * mu[k]) * (d[0][0][k] + d[1][1][k])
            trace = lam * (d[0][0] + d[1][1] + d[2][2])
            for i in range(3):
                f[3 + i][inner] += dt * (trace + 2 * mu * d[i][i])
            sxy[inner] += dt * self.mu_xy * (d[0][1] + d[1][0])
            syz[inner] += dt * self.mu_yz * (d[1][2] + d[2][1])
            sxz[inner] += dt * self.mu_xz * (d[0][2] + d[2][0])
            if top:
                szz[4, 4:-4, 4:-4] = 0
            if self.c["source"] == "explosion":
                for (dz, dy, dx), value in self._source((step + 0.5) * dt).items():
                    z, y, x = sz + dz, sy + dy, sx + dx
                    if all(4 <= i < n - 4 for i, n in zip((z, y, x), self.n)):
                        for i in (3, 4, 5):
                            f[i][z, y, x] += value
            if self.c["walls"]:
                self._images(False)
            if after is not None:
                after(step)
        if top:
            self._images(False)

    def sample(self):
        r = torch.from_numpy(_receivers3d(self.c)).cuda().long()
        x, y, z = r[:, 0] + self.ox, r[:, 1] + self.oy, r[:, 2] + self.oz
        vx, vy, vz = self.f[:3]
        return torch.stack([0.5 * (vx[z, y, x] + vx[z, y, x - 1]), 0.5 * (vy[z, y, x] + vy[z, y - 1, x]),
                            0.5 * (vz[z, y, x] + vz[z - 1, y, x])], dim=-1)

    def shot(self, first):
        n, stride, taken = self.c["steps"], self.c["stride"], []
        most = max(1, n // stride)

        def after(step):
            if (step + 1) % stride == 0 and len(taken) < most:
                taken.append(self.sample())

        self.steps(first, n, after)
        return {"gather": torch.stack(taken) if taken else None, **self.named()}

    def views(self):
        """Slices and the bounded volume of (wave, material), as the display samples them."""
        c, p = self.c, self.p
        vx, vy, vz, sxx, syy, szz = self.f[:6]

        def wave():
            def mean(f, axis):
                return 0.5 * (f + torch.roll(f, 1, 2 - axis))

            k = c["component"]
            if k == 4:
                return -(sxx + syy + szz) / 3
            v = [mean(vx, 0), mean(vy, 1), mean(vz, 2)]
            return torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2) if k == 3 else v[(2, 0, 1)[k]]

        k = c["material"]
        material = (torch.sqrt((self.lam + 2 * self.mu) * self.b) if k == 5 else
                    torch.sqrt(self.mu * self.b) if k == 6 else 1 / self.b)
        own = slice(4, -4)
        at = (c["nx"] // 2 + self.ox, c["ny"] // 2 + self.oy, c["nz"] // 3 + self.oz)
        out = []
        for a in (wave(), material):
            inner = a[own, own, own]
            parts = [a[own, at[1], own].reshape(-1), a[own, own, at[0]].reshape(-1), a[at[2], own, own].reshape(-1)]
            for axis in range(3):
                n = inner.shape[axis]
                m = min(256, n)
                x = (torch.arange(m, device="cuda", dtype=torch.float64) + 0.5) * n / m - 0.5
                i = torch.clamp(torch.floor(x).long(), 0, n - 1)
                w = (x - i).reshape([-1 if b == axis else 1 for b in range(3)])
                inner = inner.index_select(axis, i) * (1 - w) + inner.index_select(axis, torch.clamp(i + 1, max=n - 1)) * w
            out.append(torch.cat(parts + [inner.reshape(-1)]))
        return {"wave": out[0], "material": out[1]}


def _exact2d(c, seed):
    """The 2-D split-field, hybrid and free-surface schemes in float64."""
    a = _arrays2d(c, seed)
    nx, nz, npml, flag = c["nx"], c["nz"], c["npml"], c["flag"]
    free, hybrid = flag == 3 and c["up"], flag == 2
    fs, dt = npml, a["dt"]
    inv_dt = 1.0 / dt
    w = [float(v) for v in a["weights"]]

    def volume(n):
        return torch.from_numpy(a[n]).cuda().double().reshape(nz, nx)

    rho, mu, lam, l2m = (volume(n) for n in ("rho", "mu", "lambda_", "lambda2mu"))
    dx, dxh = (torch.from_numpy(a[n]).cuda().double()[4:-4].reshape(1, -1) for n in ("dx", "dx_half"))
    dz, dzh = (torch.from_numpy(a[n]).cuda().double().reshape(-1, 1) for n in ("dz", "dz_half"))
    dp = torch.from_numpy(a["dp_flat"]).cuda().double()[4:-4]
    if free:
        dz, dzh = dz.clone(), dzh.clone()
        dz[:fs + 6] = 0
        dzh[:fs + 6] = 0
    f = {n: v.double() for n, v in _initial2d(c, seed).items()}
    if hybrid:
        first = _initial2d(c, seed)
        for k, n in enumerate(TOTALS_2D):
            f[n] = (first[FIELDS_2D[2 * k]] + first[FIELDS_2D[2 * k + 1]]).double()

    def total(n):
        return f[TOTALS_2D[("vx", "vz", "sxx", "szz", "sxz").index(n)]] if hybrid else f[n + "_1"] + f[n + "_2"]

    def d(t, axis, forward, r0, taps=4):
        """Derivative of `t` on rows r0 .. nz-5 and columns 4 .. nx-5; axis 0 = x, 1 = z."""
        at = 1 if forward else 0

        def s(k):
            i, j = (r0, 4 + k) if axis == 0 else (r0 + k, 4)
            return t[i:i + nz - 4 - r0, j:j + nx - 8]

        return sum(w[r] * (s(at + r) - s(at - 1 - r)) for r in range(taps))

    def cells(t, r0, di=0, dj=0):
        return t[r0 + di:nz - 4 + di, 4 + dj:nx - 4 + dj]

    def damp(t, r0):
        return t[r0:nz - 4]

    def split(n, r0, damping, term):
        v = f[n][r0:nz - 4, 4:-4]
        v.copy_((v * (inv_dt - damping) + term) / (inv_dt + damping))

    pml = torch.ones((nz, nx), dtype=torch.bool, device="cuda")
    if npml:
        pml[npml:nz - npml, npml:nx - npml] = False
    else:
        pml[:] = False

    def stress_split():
        r0 = fs if free else 4
        vx, vz = total("vx"), total("vz")
        x_, z_ = d(vx, 0, True, r0), d(vz, 1, False, r0)
        zx, xz = d(vz, 0, False, r0), d(vx, 1, True, r0)
        if free:
            zx[0], xz[0] = d(vz, 0, False, r0, 2)[0], d(vx, 1, True, r0, 2)[0]
        l2, lm = 0.5 * (cells(l2m, r0) + cells(l2m, r0, 0, 1)), 0.5 * (cells(lam, r0) + cells(lam, r0, 0, 1))
        m = 0.5 * (cells(mu, r0) + cells(mu, r0, 1, 0))
        z, zh = damp(dz, r0), damp(dzh, r0)
        sxx1 = l2 * x_
        if free:
            sxx1[0] = dp * x_[0]
        split("sxx_1", r0, dxh, sxx1)
        split("sxx_2", r0, z, lm * z_)
        split("szz_1", r0, dxh, lm * x_)
        split("szz_2", r0, z, l2 * z_)
        split("sxz_1", r0, dx, m * zx)
        split("sxz_2", r0, zh, m * xz)
        if free:
            q = slice(4, -4)
            for n in ("sxx_2", "szz_1", "szz_2"):
                f[n][fs, q] = 0
            for k in range(1, 5):
                for n in ("szz_1", "szz_2"):
                    f[n][fs - k, q] = -f[n][fs + k, q]
                for n in ("sxz_1", "sxz_2"):
                    f[n][fs - k, q] = -f[n][fs + k - 1, q]

    def velocity_split():
        r0 = max(fs, 4) if free else 4
        sxx, szz, sxz = total("sxx"), total("szz"), total("sxz")
        z, zh = damp(dz, r0), damp(dzh, r0)
        r = cells(rho, r0)
        ra = 0.25 * (r + cells(rho, r0, 0, 1) + cells(rho, r0, 1, 0) + cells(rho, r0, 1, 1))
        if free:
            for n in FIELDS_2D[:4]:
                f[n][4:fs, 4:-4] = 0
        split("vx_1", r0, dx, d(sxx, 0, False, r0) / r)
        split("vx_2", r0, z, d(sxz, 1, False, r0) / r)
        split("vz_1", r0, dxh, d(sxz, 0, True, r0) / ra)
        split("vz_2", r0, zh, d(szz, 1, True, r0) / ra)
        for n in FIELDS_2D[:4]:
            ring(f[n])

    def ring(t):
        t[0] = t[-1] = 0
        t[:, 0] = t[:, -1] = 0

    inside = pml[4:-4, 4:-4]

    def hybrid_update(pairs):
        """(total, half 1, damping 1, term 1, half 2, damping 2, term 2) of one update."""
        for name, h1, d1, t1, h2, d2, t2 in pairs:
            t, p1, p2 = (f[n][4:-4, 4:-4] for n in (name, h1, h2))
            q1 = (p1 * (inv_dt - d1) + t1) / (inv_dt + d1)
            q2 = (p2 * (inv_dt - d2) + t2) / (inv_dt + d2)
            plain = t + dt * (t1 + t2)
            t.copy_(torch.where(inside, q1 + q2, plain))
            p1.copy_(torch.where(inside, q1, p1))
            p2.copy_(torch.where(inside, q2, p2))

    def stress_hybrid():
        vx, vz = f["vx"], f["vz"]
        x_, z_, zx, xz = d(vx, 0, True, 4), d(vz, 1, False, 4), d(vz, 0, False, 4), d(vx, 1, True, 4)
        l2, lm = 0.5 * (cells(l2m, 4) + cells(l2m, 4, 0, 1)), 0.5 * (cells(lam, 4) + cells(lam, 4, 0, 1))
        m = 0.5 * (cells(mu, 4) + cells(mu, 4, 1, 0))
        z, zh = damp(dz, 4), damp(dzh, 4)
        hybrid_update([("sigmaxz", "sxz_1", dx, m * zx, "sxz_2", zh, m * xz),
                       ("sigmaxx", "sxx_1", dxh, l2 * x_, "sxx_2", z, lm * z_),
                       ("sigmazz", "szz_1", dxh, lm * x_, "szz_2", z, l2 * z_)])

    def velocity_hybrid():
        sxx, szz, sxz = f["sigmaxx"], f["sigmazz"], f["sigmaxz"]
        z, zh = damp(dz, 4), damp(dzh, 4)
        r = cells(rho, 4)
        ra = 0.25 * (r + cells(rho, 4, 0, 1) + cells(rho, 4, 1, 0) + cells(rho, 4, 1, 1))
        hybrid_update([("vz", "vz_1", dxh, d(sxz, 0, True, 4) / ra, "vz_2", zh, d(szz, 1, True, 4) / ra),
                       ("vx", "vx_1", dx, d(sxx, 0, False, 4) / r, "vx_2", z, d(sxz, 1, False, 4) / r)])
        ring(f["vx"])
        ring(f["vz"])

    def inject(value, x, z):
        if not (4 <= x < nx - 4 and 4 <= z < nz - 4) or (free and z <= fs):
            return
        kind, one = c["type"], 1.0 if hybrid else 0.5
        if kind in (capi2d.EXPLOSIVE, capi2d.SHEAR):
            names = ("sxx", "szz") if kind == capi2d.EXPLOSIVE else ("sxz",)
            for n in names:
                for target in ((TOTALS_2D[("vx", "vz", "sxx", "szz", "sxz").index(n)],) if hybrid else (n + "_1", n + "_2")):
                    f[target][z, x] += one * value
            return
        angle = math.radians(30.0)
        force = (math.sin(angle) * value, math.cos(angle) * value) if kind == capi2d.ROTATED_FORCE else (value, value)
        if kind != capi2d.VERTICAL_FORCE:
            f["vx" if hybrid else "vx_1"][z, x] += force[0] * dt / rho[z, x]
        if kind != capi2d.HORIZONTAL_FORCE:
            mean = 0.25 * (rho[z, x] + rho[z, x + 1] + rho[z + 1, x] + rho[z + 1, x + 1])
            f["vz" if hybrid else "vz_1"][z, x] += force[1] * dt / mean

    steps, stride = c.get("steps", 1), c.get("stride", 1)
    first = _first_step(dt, 1.2 * a["f0"], steps)
    sources = [list(s) for s in _sources2d(c, a)]
    rcv = torch.from_numpy(a["rcv"]).cuda().long()
    traces = []
    sx, sz = a["src"]
    for k in range(steps):
        stress_hybrid() if hybrid else stress_split()
        velocity_hybrid() if hybrid else velocity_split()
        if not sources:
            if first + k < a["nt"]:
                inject(float(a["wavelet"][first + k]) * 1e7, sx, max(sz, fs + 1) if free else sz)
        for s in sources:
            s[1] += dt
            peak = 1.0 / s[2]
            if s[1] <= 2.5 * peak:
                x = math.pi * s[2] * (s[1] - peak)
                inject(s[3] * (1 - 2 * x * x) * math.exp(-x * x) * 1e7, s[0] % nx, s[0] // nx)
        if k % stride == 0:
            traces.append((total("vx").reshape(-1)[rcv], total("vz").reshape(-1)[rcv]))
    out = dict(f)
    if c["kind"] == "live2d":
        out.update(receivers_vx=traces[0][0], receivers_vz=traces[0][1])
    else:
        out.update(trace_vx=torch.stack([t[0] for t in traces], dim=1), trace_vz=torch.stack([t[1] for t in traces], dim=1))
    return out
