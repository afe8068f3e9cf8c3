"""Cases of the solver's real use, for timing and for comparing outputs.

A case is one call sequence of a user's program on a handle that the program
keeps: advance the simulation by a number of steps and read what it produced
(the density field as a frame, the receivers' series), or evaluate one gradient
of the receiver misfit.  Geometry, sources and receivers are made from the
seed.  `exact` is the same computation in FP64 with plain torch operations.

kind   "forward"  the family-B step: open box or ground plane, box buildings,
                  point sources, FP32 or FP16 storage
       "gradient" lbm_adjoint_grad of the receiver misfit
       "mirror" / "doppler" / "pulse" / "columns"
                  the family-A programs 02 / 03 / 01 / 04
calls  "batch"    Solver.step(n), replayed as CUDA graphs
       "single"   the reference's own loop body, one call per operation
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                     "city-scale-nlos-acoustic-engine-code_b200")
if _ROOT not in sys.path:
    sys.path.insert(0, _ROOT)

from nlos_lbm import abi, solver, workloads  # noqa: E402

CS = abi.CS
F, W, P = abi.LBM_BC_NSCBC, abi.LBM_BC_WALL, abi.LBM_BC_PERIODIC


def _fwd(name, nx, ny, nz, steps, **kw):
    c = dict(name=name, kind="forward", nx=nx, ny=ny, nz=nz, steps=steps, storage="f32", calls="batch", ground=True,
             buildings=True, pitch=32, nsrc=1, wave="sine", inject="trilinear", mach=0.0, nprobe=8, sponge=8,
             tau=0.52, frame=True, series=True)
    c.update(kw)
    return c


def listed():
    return [
        # the reference's own loop body on a small box (48x32x30, Gaussian stencil): an
        # interactive program or a caller's own schedule, five steps then a frame
        _fwd("single_calls_48", 48, 32, 30, 5, calls="single", pitch=16, inject="gauss", nprobe=4, tau=0.55,
             series=False),
        # a street block at odd sizes between two frames (parameter studies of many small runs)
        _fwd("block_97x83x41", 97, 83, 41, 200, pitch=24, nsrc=2, nprobe=12, sponge=10, tau=0.51, series=False),
        # the 128^3 acoustic scattering box, open on all faces, Gaussian stencil, FP32
        _fwd("scatter_128_f32", 128, 128, 128, 400, ground=False, pitch=64, inject="gauss", sponge=20, tau=0.55),
        # the same in FP16 storage, receivers only
        _fwd("scatter_128_f16", 128, 128, 128, 1000, storage="f16", ground=False, pitch=64, inject="gauss",
             sponge=20, tau=0.55, frame=False),
        # Lloyd's mirror 256x128x128: ground plane, no buildings, source flying at Mach 0.1
        _fwd("lloyd_256x128x128", 256, 128, 128, 200, buildings=False, mach=0.1, nprobe=64, sponge=16),
        # a city district 512x512x128 with frames, FP32
        _fwd("city_512_f32", 512, 512, 128, 200, pitch=48, nsrc=2, nprobe=64, sponge=32, tau=0.51),
        # the 1024x1024x256 city in FP16, receivers only: the largest runs
        _fwd("city_1024_f16", 1024, 1024, 256, 100, storage="f16", pitch=48, nsrc=4, nprobe=256, sponge=32,
             tau=0.51, frame=False),
        # source localisation: one gradient evaluation of its iterations, small and usual patch
        dict(name="gradient_128", kind="gradient", nx=128, ny=128, nz=128, steps=150, nprobe=64, pitch=48, sponge=16,
             tau=0.52, outer=0),
        dict(name="gradient_256", kind="gradient", nx=256, ny=256, nz=128, steps=300, nprobe=64, pitch=48, sponge=16,
             tau=0.52, outer=0),
        # 01 at its own size (its 402 steps from the pulse), 03 at half its size, 04 at its own size
        dict(name="pulse_320x320x8", kind="pulse", scale=1.0, steps=402, series=True),
        dict(name="doppler_200x200x300", kind="doppler", scale=0.5, steps=100, series=True),
        dict(name="columns_208", kind="columns", scale=1.0, steps=100, series=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward"] * 6 + ["gradient"] * 2 + ["mirror", "doppler", "pulse", "columns"])
    if kind == "forward":
        f16 = rng.random() < 0.4
        nx, ny = _log_int(rng, 24, 900), _log_int(rng, 24, 900)
        nz = _log_int(rng, 24, 200)
        cells = nx * ny * nz
        single = cells < 4_000_000 and rng.random() < 0.25
        steps = max(4, min(400, int(rng.uniform(0.5, 1.5) * 1.2e9 / cells)))
        return _fwd("", nx, ny, nz, rng.randint(3, 9) if single else steps,
                    storage="f16" if f16 else "f32", calls="single" if single else "batch",
                    ground=rng.random() < 0.7, buildings=rng.random() < 0.75, pitch=rng.choice([16, 24, 32, 48]),
                    nsrc=rng.randint(1, 4), wave=rng.choice(["sine", "ricker"]),
                    inject=rng.choice(["trilinear", "gauss"]), mach=rng.choice([0.0, 0.0, 0.1, 0.15]),
                    nprobe=rng.choice([1, 5, 16, 64, 200]), sponge=rng.choice([0, 6, 8, 10]),
                    tau=rng.choice([0.51, 0.52, 0.55]), frame=not f16, series=f16 or cells > 1_000_000)
    if kind == "gradient":
        nx, ny, nz = _log_int(rng, 40, 300), _log_int(rng, 40, 300), _log_int(rng, 32, 140)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=max(20, min(300, int(4e8 / (nx * ny * nz)))),
                    nprobe=rng.choice([1, 7, 64]), pitch=rng.choice([16, 24, 48]), sponge=rng.choice([6, 8, 16]),
                    tau=rng.choice([0.51, 0.52, 0.55]), outer=rng.choice([0, 0, 16]))
    scale = round(rng.uniform(0.2, {"mirror": 0.6, "doppler": 0.55, "pulse": 1.3, "columns": 1.1}[kind]), 3)
    return dict(kind=kind, scale=scale, steps=rng.randint(20, 100), series=True)


# ---------------------------------------------------------------- inputs

def _buildings(rng, nx, ny, nz, pitch):
    """Boxes (x0, y0, x1, y1, h) on a street grid of the given pitch; streets of >= 6 cells between them."""
    out = []
    for py in range(0, ny - pitch + 1, pitch):
        for px in range(0, nx - pitch + 1, pitch):
            a, b = 3 + rng.integers(0, 3, 2), pitch - 3 - rng.integers(0, pitch // 4, 2)
            out.append((px + a[0], py + a[1], px + b[0], py + b[1], rng.integers(4, max(6, min(80, nz * 2 // 3)))))
    return np.array(out, dtype=np.int64).reshape(-1, 5)


def _cube(cell, nx, ny, nz):
    """The single rigid cube of the scattering box, in the middle, at the height of the middle."""
    c = (nx // 2, ny // 2)
    return np.array([[c[0] - cell, c[1] - cell, c[0] + cell, c[1] + cell, nz // 2 + cell]], dtype=np.int64)


def _triangles(boxes):
    """12 triangles per box, ground to roof, 9 floats each."""
    q = np.array([(0, 3, 2), (0, 2, 1), (4, 5, 6), (4, 6, 7), (0, 1, 5), (0, 5, 4), (1, 2, 6), (1, 6, 5), (2, 3, 7),
                  (2, 7, 6), (3, 0, 4), (3, 4, 7)])
    x0, y0, x1, y1, h = boxes.T.astype(np.float64)
    z = np.zeros_like(h)
    v = np.stack([np.stack(p, 1) for p in ((x0, y0, z), (x1, y0, z), (x1, y1, z), (x0, y1, z), (x0, y0, h),
                                          (x1, y0, h), (x1, y1, h), (x0, y1, h))], 1)
    return np.ascontiguousarray(v[:, q].reshape(-1, 9), dtype=np.float32)


def _free_points(rng, n, boxes, lo, hi, near=None, spread=None):
    """n points in [lo, hi] that keep 1.5 cells off every building, around `near` where given."""
    out = []
    lo, hi = np.asarray(lo, float), np.asarray(hi, float)
    for tries in range(100000):
        if near is None:
            p = rng.uniform(lo, hi)
        else:
            p = np.clip(near + rng.normal(0, spread, 3), lo, hi)
        ok = not len(boxes) or not np.any((p[0] > boxes[:, 0] - 1.5) & (p[0] < boxes[:, 2] + 1.5) &
                                          (p[1] > boxes[:, 1] - 1.5) & (p[1] < boxes[:, 3] + 1.5) &
                                          (p[2] < boxes[:, 4] + 1.5))
        if ok:
            out.append(p)
            if len(out) == n:
                return np.array(out)
    raise RuntimeError("no free place for the points")


def _scene(case, seed):
    """What a forward or gradient case has in hand: configuration values, boxes, sources, receivers."""
    rng = np.random.default_rng([seed, case["nx"], case["ny"], case["nz"]])
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ground = case.get("ground", True)
    if not case.get("buildings", True):
        boxes = np.zeros((0, 5), np.int64)
    elif case["pitch"] >= 64:
        boxes = _cube(8, nx, ny, nz)
    else:
        boxes = _buildings(rng, nx, ny, nz, case["pitch"])
    m = 3.2
    top = max(m + 1.0, min(nz - m, nz * 0.5 if ground else nz - m))
    lo, hi = (m, m, m if not ground else 1.6), (nx - m, ny - m, top)
    nsrc = case.get("nsrc", 1)
    centre = np.array([nx * 0.5, ny * 0.5, min(top, 4.0) if ground else nz * 0.5])
    start = _free_points(rng, nsrc, boxes, lo, hi, near=centre, spread=min(12.0, nx / 5, ny / 5))
    end = start + rng.uniform(-0.2, 0.2, start.shape) * np.array([nx, ny, 0.0])
    end = np.clip(end, lo, hi)
    probes = _free_points(rng, case["nprobe"], boxes, lo, hi, near=start[0], spread=min(25.0, nx / 4, ny / 4))
    amp = 1e-3
    freq = rng.uniform(1 / 48, 1 / 24, nsrc)
    return dict(boxes=boxes, start=start, end=end, probes=probes, amp=amp, freq=freq, ground=ground,
                faces=(F, F, F, F, W if ground else F, F), sponge_faces=abi_faces(ground),
                sponge=float(case["sponge"]), strength=0.35, tau=case["tau"])


def abi_faces(ground):
    return workloads.FIVE_FACES if ground else workloads.ALL_FACES


def _forward_source(case, sc, i):
    mach = case.get("mach", 0.0)
    e = sc["end"][i] if mach > 0 else sc["start"][i]
    s = sc["start"][i]
    ricker = case.get("wave", "sine") == "ricker" or case["kind"] == "gradient"
    return dict(sx=s[0], sy=s[1], sz=s[2], ex=e[0], ey=e[1], ez=e[2], speed=mach * CS, amp=sc["amp"],
                freq=sc["freq"][i], t0=1.1 / sc["freq"][i],
                waveform=abi.LBM_WAVE_RICKER if ricker else abi.LBM_WAVE_SINE,
                injection=abi.LBM_INJECT_GAUSS if case.get("inject") == "gauss" else abi.LBM_INJECT_TRILINEAR)


def _config(case, sc):
    f16 = case.get("storage") == "f16"
    return workloads.lattice_config(case["nx"], case["ny"], case["nz"], sc["tau"], face_bc=sc["faces"],
                                    sponge_faces=sc["sponge_faces"], sponge_width=sc["sponge"],
                                    sponge_strength=sc["strength"],
                                    storage=abi.LBM_STORE_F16 if f16 else abi.LBM_STORE_F32,
                                    f16_scale=workloads.F16_HEADROOM / sc["amp"])


def _observed(case, sc):
    """Receiver series a trial source is fitted to: free-field arrivals of a source a few cells away."""
    true = sc["start"][0] + np.array([2.4, -1.6, 0.8])
    r = np.maximum(1.0, np.linalg.norm(sc["probes"] - true, axis=1))
    t = np.arange(case["steps"])[:, None] - r[None, :] / CS
    a = (math.pi * sc["freq"][0] * (t - 1.1 / sc["freq"][0])) ** 2
    return sc["amp"] * 0.05 * (1 - 2 * a) * np.exp(-a) / r[None, :]


def _family_a(case, seed):
    """The family-A programs' set-ups at a scale of their grids; source strength, period and position from the seed."""
    rng = np.random.default_rng([seed, 77])
    s, kind = case["scale"], case["kind"]
    amp, wob = rng.uniform(0.7, 1.3), rng.uniform(0.8, 1.25)
    if kind == "mirror":      # 02: ground layer, tau ramp, time-harmonic Gaussian source
        dx, n = 0.4, [max(24, int(250 * s)), max(24, int(250 * s)), max(20, int(150 * s))]
        cfg = workloads.lattice_config(*n, 0.51, x_max=n[0] * dx, y_max=n[1] * dx, z_max=n[2] * dx, dx=dx, c_phys=1.0,
                                       face_bc=(abi.LBM_BC_REST,) * 6,
                                       sponge_faces=workloads.ALL_FACES & ~(1 << abi.FACE_ZLO),
                                       sponge_width=10.0, scheme=abi.LBM_SCHEME_A, tau_sponge_max=1.0,
                                       dt=0.577350269 * dx)
        solid = np.zeros((n[2] + 2, n[1] + 2, n[0] + 2), np.uint8)
        solid[1] = 1
        ctr = [n[0] * dx * rng.uniform(0.45, 0.55), n[1] * dx * rng.uniform(0.45, 0.55), 8 * dx]
        src = dict(amp=0.5 * amp, freq=wob / 30.0, sigma=math.sqrt(1 / math.log(2.0)) / dx, mode=abi.LBM_FIELD_DST)
    elif kind == "doppler":   # 03: Mach 0.2 flow along z, zero-gradient halos, forcing
        dx = 0.25
        n = [max(24, int(400 * s)), max(24, int(400 * s)), max(24, int(600 * s))]
        cfg = workloads.lattice_config(*n, 0.51, x_max=n[0] * dx, y_max=n[1] * dx, z_max=n[2] * dx, dx=dx, c_phys=1.0,
                                       face_bc=(abi.LBM_BC_COPY,) * 6, sponge_faces=workloads.ALL_FACES,
                                       sponge_width=min(20.0, min(n) // 3), scheme=abi.LBM_SCHEME_A,
                                       tau_sponge_max=0.9, flow=(0.0, 0.0, 0.2 * CS), dt=CS * dx)
        solid = None
        ctr = [m * dx * rng.uniform(0.45, 0.55) for m in n]
        src = dict(amp=0.01 * amp, freq=wob / (30.0 * CS * dx), sigma=1.0, mode=abi.LBM_FIELD_FORCE)
    elif kind == "pulse":     # 01: initial pulse, cylinder, destination blend, periodic z
        dx, n0 = 0.05, max(40, int(320 * s))
        n = [n0, n0, max(3, int(8 * s))]
        half = n0 * dx / 2
        side = sum(1 << f for f in (abi.FACE_XLO, abi.FACE_XHI, abi.FACE_YLO, abi.FACE_YHI))
        cfg = workloads.lattice_config(*n, 0.505, x_min=-half, x_max=half, y_min=-half, y_max=half, z_max=n[2] * dx,
                                       dx=dx, c_phys=1.0, face_bc=(abi.LBM_BC_REST,) * 4 + (P, P), sponge_faces=side,
                                       sponge_width=10.0, sponge_strength=1.0, sponge_blend=1,
                                       scheme=abi.LBM_SCHEME_A, dt=math.sqrt(1 / 3) * dx)
        c = -half + (np.arange(-1, n0 + 1) + 0.5) * dx
        solid = np.broadcast_to((c[None, :] ** 2 + c[:, None] ** 2) < 0.25, (n[2] + 2, n0 + 2, n0 + 2))
        pc = half * np.array([rng.uniform(0.3, 0.6), rng.uniform(-0.2, 0.2)])
        pulse = 0.01 * amp * np.exp(-math.log(2.0) * wob * ((c[None, :] - pc[0]) ** 2 + (c[:, None] - pc[1]) ** 2))
        rho0 = np.where(solid[0], 0.0, pulse)[1:-1, 1:-1]
        src, ctr = None, None
    else:                     # 04: cylinder, radial blend layer, line source before the step, periodic z
        n0 = max(40, int(208 * s))
        n, dx = [n0] * 3, 26.0 / n0
        cfg = workloads.lattice_config(*n, 0.51, x_min=-13.0, x_max=13.0, y_min=-13.0, y_max=13.0, z_min=-13.0,
                                       z_max=13.0, dx=dx, c_phys=1.0, face_bc=(abi.LBM_BC_REST,) * 4 + (P, P),
                                       sponge_faces=0, sponge_width=0.0, sponge_blend=1, scheme=abi.LBM_SCHEME_A,
                                       dt=0.577350269 * dx)
        ctr = [0.0, rng.uniform(-7.0, -5.0), 0.0]
        solid2, blend, weight = workloads.hpc_columns(dx, -13.0, n0, src_y=ctr[1])
        solid = np.broadcast_to(solid2, (n0 + 2,) + solid2.shape)
        src = dict(amp=0.01 * amp, freq=wob / (30.0 * 0.577350269 * dx), sigma=1.0, mode=abi.LBM_FIELD_PRE)
    lo = np.array([cfg.x_min, cfg.y_min, cfg.z_min])
    probes = lo + np.stack([rng.uniform(0.15, 0.85, 64) * m * cfg.dx for m in n], 1)
    d = dict(cfg=cfg, n=n, solid=None if solid is None else np.ascontiguousarray(solid, dtype=np.uint8),
             probes=probes, src=src, ctr=ctr, blend=None, weight=None, rho0=None)
    if kind == "pulse":
        d["rho0"] = np.ascontiguousarray(np.broadcast_to(rho0, (n[2], n[1], n[0])))
    if kind == "columns":
        d["blend"], d["weight"] = blend, weight
    return d


def prepare(case, seed):
    if case["kind"] in ("forward", "gradient"):
        sc = _scene(case, seed)
        srcs = [abi.reference_source(**_forward_source(case, sc, i)) for i in range(len(sc["start"]))]
        s = solver.Solver(_config(case, sc), srcs, sc["probes"],
                          triangles=_triangles(sc["boxes"]) if len(sc["boxes"]) else None)
        st = dict(case=case, solver=s, scale=workloads.F16_HEADROOM / sc["amp"])
        if case["kind"] == "gradient":
            st["observed"] = _observed(case, sc)
        return st
    a = _family_a(case, seed)
    srcs = []
    if a["src"]:
        x, y, z = a["ctr"]
        srcs = [abi.reference_source(sx=x, sy=y, sz=z, ex=x, ey=y, ez=z, amp=a["src"]["amp"], freq=a["src"]["freq"],
                                     waveform=abi.LBM_WAVE_SINE, injection=abi.LBM_INJECT_FIELD,
                                     sigma_cells=a["src"]["sigma"], field_mode=a["src"]["mode"])]
    s = solver.Solver(a["cfg"], srcs, a["probes"], mask=None if a["solid"] is None else a["solid"].ravel(),
                      blend_xy=a["blend"], field_xy=a["weight"])
    if a["rho0"] is not None:
        s.set_density(a["rho0"])
    return dict(case=case, solver=s)


# ---------------------------------------------------------------- one pass

def run(state):
    """Fields and series are kept in the type that the storage carries: the library hands series, energies and
    gradients over as doubles that hold results of FP32 arithmetic on FP32 or (scaled) FP16 state."""
    c, s = state["case"], state["solver"]
    if c["kind"] == "gradient":
        loss, gpos, gsig, pred = s.adjoint_grad(state["observed"], ckpt_outer=c["outer"])
        return {"loss": np.float32(loss), "grad_pos": gpos.astype(np.float32), "grad_signal": gsig.astype(np.float32),
                "predicted": pred.astype(np.float32)}
    if c.get("calls") == "single":
        for _ in range(c["steps"]):
            s.apply_source(s.step_count * s.dt)
            s.exchange_halos()
            s.step_collision_bgk()
            s.record_probes()
    else:
        s.step(c["steps"])
    out = {}
    if c.get("frame", True):
        out["rho"] = s.get_rho()
    if c["series"]:
        p = s.get_probes()
        out["series"] = (p * state["scale"]).astype(np.float16) if c.get("storage") == "f16" else p.astype(np.float32)
    else:
        out["energy"] = s.get_probe_energy().astype(np.float32)
    return out


def _cells(case):
    if case["kind"] in ("forward", "gradient"):
        return case["nx"] * case["ny"] * case["nz"]
    s = case["scale"]
    if case["kind"] == "mirror":
        return max(24, int(250 * s)) ** 2 * max(20, int(150 * s))
    if case["kind"] == "doppler":
        return max(24, int(400 * s)) ** 2 * max(24, int(600 * s))
    if case["kind"] == "pulse":
        return max(40, int(320 * s)) ** 2 * max(3, int(8 * s))
    return max(40, int(208 * s)) ** 3


def work(case):
    """A step reads and writes the 19 populations of every cell once; a gradient does so forward and backward.
    About 250 operations a cell and step (moments, equilibrium, relaxation, sponge)."""
    n, t = _cells(case), case["steps"]
    size = 2 if case.get("storage") == "f16" else 4
    passes = 2 if case["kind"] == "gradient" else 1
    frame = 4 * n if case["kind"] != "gradient" and case.get("frame", True) else 0
    return {"bytes": float(passes * n * t * 2 * 19 * size + frame), "flops": float(passes * n * t * 250)}


# ---------------------------------------------------------------- FP64 restatement in torch

EX, EY, EZ, WQ = abi.EX, abi.EY, abi.EZ, abi.W
INV = [next(p for p in range(19) if (EX[p], EY[p], EZ[p]) == (-EX[q], -EY[q], -EZ[q])) for q in range(19)]


def _sl(v, q, nx, ny, nz):
    """Interior-sized view of a halo-inclusive [z, y, x] array at the cells that direction q comes from."""
    return v[..., 1 - EZ[q]:1 - EZ[q] + nz, 1 - EY[q]:1 - EY[q] + ny, 1 - EX[q]:1 - EX[q] + nx]


def _moments(g):
    r, jx, jy, jz = g[0], 0, 0, 0
    for q in range(1, 19):
        r = r + g[q]
        jx = jx + EX[q] * g[q] if EX[q] else jx
        jy = jy + EY[q] * g[q] if EY[q] else jy
        jz = jz + EZ[q] * g[q] if EZ[q] else jz
    return r, jx, jy, jz


def _geq(q, rp, r, ux, uy, uz, u2):
    """feq - w of density r = 1 + rp and velocity u."""
    cu = EX[q] * ux + EY[q] * uy + EZ[q] * uz
    return WQ[q] * (rp + r * (3.0 * cu + 4.5 * cu * cu - 1.5 * u2))


def _open_ghost(g, axis, side):
    """Characteristic ghost populations from the interior layer g [19, ...] of one open face."""
    rp, jx, jy, jz = _moments(g)
    r = 1.0 + rp
    u = [jx / r, jy / r, jz / r]
    p = rp / 3.0
    w = u[axis] - p / CS if side == 0 else u[axis] + p / CS
    ub = list(u)
    ub[axis] = 0.5 * w
    rb = (-0.5 if side == 0 else 0.5) * CS * w * 3.0
    u2, ub2 = u[0] ** 2 + u[1] ** 2 + u[2] ** 2, ub[0] ** 2 + ub[1] ** 2 + ub[2] ** 2
    return torch.stack([_geq(q, rb, 1.0 + rb, *ub, ub2) + g[q] - _geq(q, rp, r, *u, u2) for q in range(19)])


def _solid_b(case, sc, dev):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    h = np.zeros((ny + 2, nx + 2))
    for x0, y0, x1, y1, top in sc["boxes"]:
        h[y0 + 1:y1 + 1, x0 + 1:x1 + 1] = np.maximum(h[y0 + 1:y1 + 1, x0 + 1:x1 + 1], top)
    z = torch.arange(-1, nz + 1, device=dev, dtype=torch.float64) + 0.5
    m = z[:, None, None] < torch.tensor(h, device=dev)[None]
    if not len(sc["boxes"]):
        m = torch.zeros_like(m)
    m[:, :, 0] = m[:, :, -1] = False
    m[:, 0, :] = m[:, -1, :] = False
    m[0] = sc["faces"][4] == W
    m[-1] = False
    return m


def _sponge_b(case, sc, dev):
    w, prof = sc["sponge"], []
    for a, n in enumerate((case["nx"], case["ny"], case["nz"])):
        x = torch.arange(n, device=dev, dtype=torch.float64) + 0.5
        d = torch.full_like(x, 1e30)
        if sc["sponge_faces"] & (1 << (2 * a)):
            d = torch.minimum(d, x)
        if sc["sponge_faces"] & (1 << (2 * a + 1)):
            d = torch.minimum(d, n - x)
        prof.append(torch.where(d < w, sc["strength"] * ((w - d) / max(w, 1e-30)) ** 2, torch.zeros_like(d)))
    return torch.maximum(prof[2][:, None, None], torch.maximum(prof[1][None, :, None], prof[0][None, None, :]))


def _path(src, t):
    s, e = (np.array([src[k + c] for c in "xyz"]) for k in "se")
    dist = float(np.linalg.norm(e - s))
    if dist < 1e-12 or src["speed"] < 1e-12:
        return s
    return s + min(1.0, t * src["speed"] / dist) * (e - s)


def _signal(src, t):
    if src["waveform"] == abi.LBM_WAVE_SINE:
        return src["amp"] * math.sin(2 * math.pi * src["freq"] * t)
    a = (math.pi * src["freq"] * (t - src["t0"])) ** 2
    return src["amp"] * (1 - 2 * a) * math.exp(-a)


def _stencil(src, pos, solid, nx, ny, nz):
    """Cells (k, j, i) of one injection and their normalised weights; differentiable in pos (a torch triple)."""
    dev = pos.device
    if src["injection"] == abi.LBM_INJECT_TRILINEAR:
        base = torch.floor(pos.detach() - 0.5)
        o = torch.tensor([(b & 1, (b >> 1) & 1, b >> 2) for b in range(8)], device=dev, dtype=torch.float64)
        t = pos - 0.5 - base
        w = torch.where(o > 0, t, 1 - t).prod(1)
    else:
        base = torch.floor(pos.detach())
        r = torch.arange(-2, 3, device=dev, dtype=torch.float64)
        o = torch.stack([v.reshape(-1) for v in torch.meshgrid(r, r, r, indexing="ij")], 1)
        w = torch.exp(-0.5 * ((base + o + 0.5 - pos) ** 2).sum(1) / 1.25 ** 2)
    c = (base + o).long()
    ok = ((c >= 0) & (c < torch.tensor([nx, ny, nz], device=dev))).all(1)
    c, w = c[ok], w[ok]
    fluid = ~solid[c[:, 2] + 1, c[:, 1] + 1, c[:, 0] + 1]
    c, w = c[fluid], w[fluid]
    return c, w / w.sum()


def _step_b(g, add, solid, sponge, faces, omega):
    """One family-B step of interior deviations g [19, z, y, x]; `add` = (cells, amounts) of the source.
    Returns the new deviations and the pulled density deviation."""
    nz, ny, nx = g.shape[1:]
    wq = torch.tensor(WQ, device=g.device, dtype=torch.float64)
    if add is not None:
        (c, amount) = add
        g = g.index_put((torch.arange(19, device=g.device)[:, None], c[None, :, 2], c[None, :, 1], c[None, :, 0]),
                        wq[:, None] * amount[None, :], accumulate=True)
    h = torch.zeros((19, nz + 2, ny + 2, nx + 2), device=g.device, dtype=torch.float64)
    h[:, 1:-1, 1:-1, 1:-1] = g
    for f, bc in enumerate(faces):
        if bc != F:
            continue
        axis, side = f // 2, f % 2
        at, to = (-1, -1) if side else (0, 0)
        if axis == 0:
            h[:, 1:-1, 1:-1, to] = _open_ghost(g[:, :, :, at], axis, side)
        elif axis == 1:
            h[:, 1:-1, to, 1:-1] = _open_ghost(g[:, :, at, :], axis, side)
        else:
            h[:, to, 1:-1, 1:-1] = _open_ghost(g[:, at], axis, side)
    p = [torch.where(_sl(solid, q, nx, ny, nz), g[INV[q]], _sl(h[q], q, nx, ny, nz)) for q in range(19)]
    rp, jx, jy, jz = _moments(p)
    r = 1.0 + rp
    ux, uy, uz = jx / r, jy / r, jz / r
    u2 = ux * ux + uy * uy + uz * uz
    keep = 1.0 - sponge
    new = torch.stack([keep * (p[q] - omega * (p[q] - _geq(q, rp, r, ux, uy, uz, u2))) for q in range(19)])
    rest = solid[1:-1, 1:-1, 1:-1]
    # a SOLID cell passes its pulled values on (an open face's ghost may be built from it)
    return torch.where(rest, torch.stack(p), new), torch.where(rest, torch.zeros_like(rp), rp)


def _read(rp, probes, lo, dx):
    i = torch.tensor(np.floor((probes - lo) / dx).astype(np.int64), device=rp.device)
    return rp[i[:, 2], i[:, 1], i[:, 0]]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _exact_forward(case, seed):
    dev, sc = _device(), _scene(case, seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    solid, sponge = _solid_b(case, sc, dev), _sponge_b(case, sc, dev)
    srcs = [_forward_source(case, sc, i) for i in range(len(sc["start"]))]
    g = torch.zeros((19, nz, ny, nx), device=dev, dtype=torch.float64)
    series = []
    for s in range(case["steps"]):
        cells, amounts = [], []
        for src in srcs:
            c, w = _stencil(src, torch.tensor(_path(src, s), device=dev), solid, nx, ny, nz)
            cells.append(c)
            amounts.append(w * _signal(src, s))
        g, rp = _step_b(g, (torch.cat(cells), torch.cat(amounts)), solid, sponge, sc["faces"], 1.0 / sc["tau"])
        series.append(_read(rp, sc["probes"], np.zeros(3), 1.0))
    series = torch.stack(series)
    out = {"rho": rp} if case.get("frame", True) else {}
    if case["series"]:
        out["series"] = series * (workloads.F16_HEADROOM / sc["amp"]) if case["storage"] == "f16" else series
    else:
        out["energy"] = (series ** 2).sum(0)
    return {k: v.cpu() for k, v in out.items()}


def _exact_gradient(case, seed):
    from torch.utils.checkpoint import checkpoint

    dev, sc = _device(), _scene(case, seed)
    nx, ny, nz, T = case["nx"], case["ny"], case["nz"], case["steps"]
    solid, sponge = _solid_b(case, sc, dev), _sponge_b(case, sc, dev)
    src = _forward_source(case, sc, 0)
    pos = torch.tensor(sc["start"][0], device=dev, requires_grad=True)
    val = torch.tensor([_signal(src, s) for s in range(T)], device=dev, dtype=torch.float64, requires_grad=True)
    observed = torch.tensor(_observed(case, sc), device=dev)
    g = torch.zeros((19, nz, ny, nx), device=dev, dtype=torch.float64)

    def one(g, pos, v):
        c, w = _stencil(src, pos, solid, nx, ny, nz)
        g, rp = _step_b(g, (c, w * v), solid, sponge, sc["faces"], 1.0 / sc["tau"])
        return g, _read(rp, sc["probes"], np.zeros(3), 1.0)

    rows = []
    for s in range(T):
        g, row = checkpoint(one, g, pos, val[s], use_reentrant=False)
        rows.append(row)
    pred = torch.stack(rows)
    loss = 0.5 * ((pred - observed) ** 2).sum()
    loss.backward()
    return {"loss": loss.detach().cpu(), "grad_pos": pos.grad.cpu(), "grad_signal": val.grad.cpu(),
            "predicted": pred.detach().cpu()}


def _exact_a(case, seed):
    dev, a = _device(), _family_a(case, seed)
    cfg, (nx, ny, nz), d = a["cfg"], a["n"], torch.float64
    tau = torch.full((nz + 2, ny + 2, nx + 2), cfg.tau, device=dev, dtype=d)
    blend = torch.zeros((nz, ny, nx), device=dev, dtype=d)
    lo, hi, n = (cfg.x_min, cfg.y_min, cfg.z_min), (cfg.x_max, cfg.y_max, cfg.z_max), (nx, ny, nz)
    dist, depth = [], []
    for ax in range(3):
        g = torch.arange(-1, n[ax] + 1, device=dev, dtype=d)
        v, dep = torch.full_like(g, 1e9), torch.zeros_like(g)
        x, th = lo[ax] + (g + 0.5) * cfg.dx, cfg.sponge_width * cfg.dx
        if cfg.sponge_faces & (1 << (2 * ax)):
            v, dep = torch.minimum(v, g), torch.maximum(dep, lo[ax] + th - x)
        if cfg.sponge_faces & (1 << (2 * ax + 1)):
            v, dep = torch.minimum(v, n[ax] - 1 - g), torch.maximum(dep, x - (hi[ax] - th))
        dist.append(v)
        depth.append(dep)

    def spread(f, p):
        return f(p[2][:, None, None], f(p[1][None, :, None], p[0][None, None, :]))

    if cfg.tau_sponge_max > 0:
        dd, w = spread(torch.minimum, dist), int(cfg.sponge_width)
        tau = torch.where((dd >= 0) & (dd < w), cfg.tau + (cfg.tau_sponge_max - cfg.tau) * ((w - dd) / w) ** 2, tau)
    if cfg.sponge_blend and cfg.sponge_width > 0:
        dd = spread(torch.maximum, [v[1:-1] for v in depth])
        blend = cfg.sponge_strength * (dd / (cfg.sponge_width * cfg.dx)) ** 2
    if a["blend"] is not None:
        blend = torch.maximum(blend, torch.tensor(a["blend"], device=dev)[None])
    blend = torch.where(blend > 1e-6, blend, torch.zeros_like(blend))
    solid = torch.zeros((nz + 2, ny + 2, nx + 2), device=dev, dtype=torch.bool)
    if a["solid"] is not None:
        solid = torch.tensor(a["solid"], device=dev) != 0
    periodic, copy = cfg.face_bc[4] == P, cfg.face_bc[0] == abi.LBM_BC_COPY
    if periodic:
        solid[0], solid[-1] = solid[-2].clone(), solid[1].clone()
    src, field = a["src"], None
    if src:
        if a["weight"] is not None:
            field = torch.nn.functional.pad(torch.tensor(a["weight"], device=dev)[None, None], (1, 1, 1, 1),
                                            mode="replicate")[0, 0].expand(nz + 2, ny + 2, nx + 2)
        else:
            x = [lo[ax] + (torch.arange(-1, n[ax] + 1, device=dev, dtype=d) + 0.5) * cfg.dx - a["ctr"][ax]
                 for ax in range(3)]
            r2 = x[2][:, None, None] ** 2 + x[1][None, :, None] ** 2 + x[0][None, None, :] ** 2
            field = torch.exp(-r2 / (2 * (src["sigma"] * cfg.dx) ** 2))
    fl = list(cfg.flow)
    f2 = sum(v * v for v in fl)
    f = torch.stack([torch.full((nz + 2, ny + 2, nx + 2), _geq(q, 0.0, 1.0, *fl, f2), device=dev, dtype=d)
                     for q in range(19)])
    inner = (slice(1, -1),) * 3
    rest = solid[inner]
    if a["rho0"] is not None:
        rp = torch.where(rest, torch.zeros_like(blend), torch.tensor(a["rho0"], device=dev))
        for q in range(19):
            f[q][inner] = _geq(q, rp, 1.0 + rp, *fl, f2)
    series = []
    for s in range(case["steps"]):
        mass = src["amp"] * math.sin(2 * math.pi * src["freq"] * s * cfg.dt) * cfg.dt if src else 0.0
        mode = src["mode"] if src else -1
        if mode == abi.LBM_FIELD_PRE:
            add = torch.where(rest, torch.zeros_like(blend), field[inner] * mass)
            for q in range(19):
                f[q][inner] += WQ[q] * add
        for h, i in ((0, 1), (-1, -2)):
            if copy:
                f[:, :, :, h] = f[:, :, :, i]
            else:
                f[:, :, :, h] = 0.0
        for h, i in ((0, 1), (-1, -2)):
            if copy:
                f[:, :, h] = f[:, :, i]
            else:
                f[:, :, h] = 0.0
        for h, i, o in ((0, 1, -2), (-1, -2, 1)):
            f[:, h] = f[:, i] if copy else f[:, o] if periodic else 0.0
        rp, jx, jy, jz = _moments(f)
        r = 1.0 + rp
        ux, uy, uz = jx / r, jy / r, jz / r
        u2 = ux * ux + uy * uy + uz * uz
        rho, new = 0, torch.empty((19, nz, ny, nx), device=dev, dtype=d)
        for q in range(19):
            c = f[q] - (f[q] - _geq(q, rp, r, ux, uy, uz, u2)) / tau
            if mode == abi.LBM_FIELD_FORCE:
                cu = EX[q] * fl[0] + EY[q] * fl[1] + EZ[q] * fl[2]
                c = c + WQ[q] * mass * (1 + 3 * cu) * field * (1 - 0.5 / tau)
            c = _sl(c, q, nx, ny, nz)
            if mode == abi.LBM_FIELD_DST:
                c = c + WQ[q] * mass * field[inner]
            new[q] = torch.where(_sl(solid, q, nx, ny, nz), f[INV[q]][inner], (1 - blend) * c)
            rho = rho + new[q]
        f[(slice(None),) + inner] = torch.where(rest, f[(slice(None),) + inner], new)
        rho = torch.where(rest, torch.zeros_like(rho), rho)
        series.append(_read(rho, a["probes"], np.array(lo), cfg.dx))
    return {"rho": rho.cpu(), "series": torch.stack(series).cpu()}


def exact(case, seed):
    n, t = _cells(case), case["steps"]
    if case["kind"] == "gradient":
        # one FP64 state per step is kept for the way back
        return _exact_gradient(case, seed) if n * t * 152 < 60e9 else None
    if n > 40_000_000 or n * t > 7_000_000_000:
        return None   # beyond some 20 seconds in FP64
    with torch.no_grad():
        return _exact_forward(case, seed) if case["kind"] == "forward" else _exact_a(case, seed)
