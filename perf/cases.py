"""Performance cases of the SPH-erosion step: the work that programs have it do.

A case is one pass through the public entry points of `sph_gb300` (the ctypes
binding of include/sph_erosion.h).  The simulation cases start from a settled,
disordered pool of fluid over rough terrain: the state that a run spends most
of its time in, once the initial block has collapsed.  The fluid's equation of
state is soft (P = k (rho - rho0)), so a settled pool is compressed towards
its bottom by exp(g depth / k); the pools are made with that profile, 30 to
100 neighbours within h of a particle.

Kinds of case:

  step     one or many scenes in one system, stepped and read back with the
           asynchronous readback into pinned memory (a headless run that keeps
           every frame)
  frame    an interactive frame of the default scene: one step, then the
           positions, at once
  record   a validation frame: ordered sums, every FluidParticle field back
  static   the allocation-free density pass on a caller's device buffer
  serve    the request server on a burst of requests
  mesh     the terrain surface's vertices and indices for a redraw
"""
from __future__ import annotations

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sph-erosion_gb300"))

import sph_gb300 as S  # noqa: E402
import workloads as W  # noqa: E402

# Kernel variants in use: the library's default (exact arithmetic, neighbour
# lists) and what the autotuner picks on every large workload (fast
# arithmetic, packed records, counter-scheduled warps).
DEFAULT, TUNED = 88, 164088


def _step(name, **kw):
    case = dict(name=name, kind="step", n=16384, scenes=1, steps=16, variant=DEFAULT, tile=256, cell_mult=1.0,
                box="cube", tw=128, td=128, valleys=False, erosion=True, terrain_back=False)
    case.update(kw)
    return case


def listed():
    return [
        # The reference's default scene, Initialize(1000) at dt = 0.01, drawn
        # frame by frame: latency of one step and one readback.
        dict(name="frame_1k", kind="frame", n=1000),
        # The validation mode on a small scene: sums in the reference's order
        # and all 27 record fields read back each step.
        dict(name="record_5k", kind="record", n=5000),
        # The plain small configuration (16,384 particles, unit box, 128 x 128
        # terrain) with the library's defaults, one captured graph per pass,
        # the eroded terrain read back for drawing.
        _step("plain_16k", n=16384, steps=16, terrain_back=True),
        # A medium scene with the defaults, nothing of it a round number.
        _step("odd_100k", n=100003, steps=4, tw=257, td=193),
        # The 1M-particle configuration (4 x 1 x 4 m, 1024 x 1024 terrain)
        # with the defaults ...
        _step("plain_1m", n=1 << 20, steps=2, box="flat", tw=1024, td=1024),
        # ... and with the kernels and cells that the autotuner picks for it.
        _step("plain_1m_tuned", n=1 << 20, steps=4, box="flat", tw=1024, td=1024, variant=TUNED, cell_mult=0.5),
        # The batched form: scenes of very uneven sizes (2,048 to 131,072
        # particles) in one system, the autotuner's pick for batches.
        _step("batch_48", n=131072, scenes=48, steps=8, tw=256, td=256, variant=TUNED),
        # The rainfall configuration once the rain has pooled in the carved
        # valleys: the largest scene, very uneven column heights.
        _step("rain_8m", n=1 << 23, steps=1, box="flat", tw=4096, td=4096, valleys=True, variant=TUNED, tile=128),
        # Density of a caller's particles, without an allocation.
        dict(name="static_20k", kind="static", n=20011),
        # The request server: a burst of small and medium requests, each run
        # to its end.
        dict(name="serve_16", kind="serve", requests=16, n=65536, steps=96, variant=TUNED),
        # Redraw of an eroded 1024 x 1024 terrain.
        dict(name="mesh_1024", kind="mesh", tw=1024, td=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same ranges: kinds by how often programs use them."""
    kind = rng.choice(["step"] * 7 + ["batch"] * 3 + ["frame", "record", "static", "serve", "mesh"])
    if kind == "step":
        n = _log(rng, 1000, 1 << 20)
        side = _log(rng, 33, 1025)
        flat = n > 150000
        case = _step("", n=n, steps=rng.choice([1, 4, 16]) if n < 200000 else rng.choice([1, 2, 3]),
                     box="flat" if flat else "cube", tw=side, td=max(2, side + rng.randint(-16, 16)),
                     variant=rng.choice([DEFAULT, TUNED]), tile=rng.choice([128, 256]),
                     cell_mult=rng.choice([1.0, 0.5]), erosion=rng.random() < 0.8, valleys=flat and rng.random() < 0.3)
    elif kind == "batch":
        case = _step("", n=_log(rng, 4096, 131072), scenes=rng.randint(8, 48), steps=rng.choice([1, 4, 8]),
                     tw=256, td=256, variant=rng.choice([DEFAULT, TUNED]), tile=rng.choice([128, 256]),
                     cell_mult=rng.choice([1.0, 0.5]))
    elif kind == "frame":
        case = dict(kind="frame", n=_log(rng, 27, 8000))
    elif kind == "record":
        case = dict(kind="record", n=_log(rng, 300, 16384))
    elif kind == "static":
        case = dict(kind="static", n=_log(rng, 100, 32768))
    elif kind == "serve":
        case = dict(kind="serve", requests=rng.randint(4, 16), n=_log(rng, 8192, 65536), steps=rng.randint(32, 96),
                    variant=rng.choice([DEFAULT, TUNED]))
    else:
        case = dict(kind="mesh", tw=_log(rng, 33, 1025), td=_log(rng, 33, 1025))
    case.pop("name", None)
    return case


# ---- inputs ------------------------------------------------------------------
SPACING, H = W.SPACING, W.H
ALPHA = -W.PHYS["gravity"][1] / W.PHYS["gas_stiffness"]  # compression of a settled pool, 1/m


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _heights(seed, w, d, amplitude, valleys):
    """Rough terrain, metres above the box floor: octaves of bilinear noise."""
    g = _gen(seed)
    out = torch.zeros(1, 1, d, w, device="cuda", dtype=torch.float64)
    amp, total = 1.0, 0.0
    for octave in range(6):
        cells = 4 << octave
        grid = torch.rand(1, 1, cells + 1, cells + 1, generator=g, device="cuda", dtype=torch.float64)
        out += amp * torch.nn.functional.interpolate(grid, size=(d, w), mode="bilinear", align_corners=True)
        total += amp
        amp *= 0.5
    f = out[0, 0] / total
    if valleys:
        f = torch.clamp(2.5 * (f - 0.5).abs(), max=1.0)  # channels where the noise crosses its middle
    return (f * amplitude).float()


def _bilinear(h, x, z, half):
    """Terrain height at x, z (box centred at 0)."""
    d, w = h.shape
    fx = ((x + half[0]) * ((w - 1) / (2 * half[0]))).clamp(0, w - 1)
    fz = ((z + half[2]) * ((d - 1) / (2 * half[2]))).clamp(0, d - 1)
    i, j = fx.long().clamp(max=w - 2), fz.long().clamp(max=d - 2)
    tx, tz = fx - i, fz - j
    flat = h.reshape(-1).double()
    at = j * w + i
    a0 = flat[at] + tx * (flat[at + 1] - flat[at])
    a1 = flat[at + w] + tx * (flat[at + w + 1] - flat[at + w])
    return a0 + tz * (a1 - a0)


def _pool(seed, n, half, heights):
    """n particles of a settled pool: horizontal lattice layers whose spacing
    shrinks with depth, jittered, cut off by the terrain; slow random motion."""
    g = _gen(seed + 1)
    area = 4.0 * half[0] * half[2]
    sample = heights.reshape(-1).double()
    if sample.numel() > 65536:
        sample = sample[:: sample.numel() // 65536]
    sample = torch.sort(sample).values.cpu().numpy()

    def layers(top):
        out, z = [], 0.5 * SPACING
        while z < top:
            s = SPACING * math.exp(-ALPHA * z / 3)
            out.append((top - z, s, area / s ** 2 * np.searchsorted(sample, top - z) / len(sample)))
            z += s
        return out

    lo, hi = 0.0, 2.0 * half[1]
    for _ in range(40):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if sum(c for _, _, c in layers(mid)) < 1.03 * n + 60 else (lo, mid)
    top = hi
    for _ in range(8):
        parts, have = [], 0
        for y, s, _ in reversed(layers(top)):  # from the bottom up
            kx, kz = max(1, int(2 * half[0] / s)), max(1, int(2 * half[2] / s))
            m = kx * kz
            i = torch.arange(m, device="cuda", dtype=torch.float64)
            r = torch.rand(3, m, generator=g, device="cuda", dtype=torch.float64) * 0.5 - 0.25
            x = -half[0] + (torch.remainder(i, kx) + 0.5) * (2 * half[0] / kx) + r[0] * s
            z = -half[2] + (torch.div(i, kx, rounding_mode="floor") + 0.5) * (2 * half[2] / kz) + r[1] * s
            p = torch.stack([x, y + r[2] * s - half[1], z], 1)
            p = p[p[:, 1] + half[1] > _bilinear(heights, x, z, half) + 0.2 * s]
            parts.append(p)
            have += len(p)
        if have >= n:
            break
        top += 0.5 * SPACING
    pos = torch.cat(parts)[:n].float()
    vel = (torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64) * 0.02).float()
    if len(pos) < n:
        raise ValueError("the box holds fewer than %d particles" % n)
    return pos, vel


def _half(n, box):
    """Half extents: the 1M configuration's floor area per particle under a
    1 m ceiling (2 m for the rainfall), or a cube a quarter full."""
    if box == "flat":
        f = 2.0 * math.sqrt(n / (1 << 20))
        return (f, 0.5 if n <= 1 << 20 else 1.0, f)
    side = max(0.2, (n * SPACING ** 3 / 0.26) ** (1 / 3))
    return (side / 2, side / 2, side / 2)


def _scenes(case):
    """(particles, terrain width, depth) of each scene of a step case: one as
    stated, or a spread of sizes, log-uniform down to 2,048."""
    m = case["scenes"]
    if m == 1:
        return [(case["n"], case["tw"], case["td"])]
    rng = np.random.default_rng(case["n"] * 64 + m)
    n = np.exp(rng.uniform(math.log(2048), math.log(case["n"]), m)).astype(int)
    side = rng.choice([64, 128, 200, case["tw"]], m)
    return [(int(a), int(b), int(b)) for a, b in zip(n, side)]


def _step_inputs(case, seed):
    """[(parameters, positions, velocities, heights)] of a step case."""
    out = []
    for k, (n, tw, td) in enumerate(_scenes(case)):
        half = _half(n, case["box"])
        prm = dict(W.PHYS, box_half=half, cell_mult=case["cell_mult"], erosion=int(case["erosion"]))
        amp = 0.5 if case["valleys"] else 0.3 if case["box"] == "flat" else 0.25 * 2 * half[1]
        h = _heights(seed + 131 * k, tw, td, amp, case["valleys"])
        pos, vel = _pool(seed + 131 * k, n, half, h)
        out.append((prm, pos, vel, h))
    return out


def _default_block(case, seed, jitter):
    """The reference's lattice block (spacing 0.025), slightly disordered."""
    side = int(math.ceil(round(case["n"] ** (1 / 3), 9)))
    k = torch.arange(side ** 3, device="cuda")
    g = _gen(seed)
    idx = torch.stack([k // (side * side), k // side % side, k % side], 1).double()
    org = torch.tensor([-0.2, -0.05, -0.15], dtype=torch.float64, device="cuda")
    r = torch.rand(side ** 3, 3, generator=g, device="cuda", dtype=torch.float64) - 0.5
    pos = (org + 0.025 * (idx + jitter * r))[: case["n"]].float()
    vel = (torch.randn(len(pos), 3, generator=g, device="cuda", dtype=torch.float64) * 0.05).float()
    half = max(0.2, 0.0125 * side + 0.08)  # the reference's box, widened for larger blocks
    return pos, vel, half


def _small_inputs(case, seed):
    """(parameters, positions, velocities) of frame, record and static cases."""
    if case["kind"] == "frame":
        pos, vel, half = _default_block(case, seed, 0.1)
        return dict(dt=0.01, box_half=(half,) * 3), pos, vel
    if case["kind"] == "record":
        # shallow enough that no particle has more neighbours than the
        # ordered mode lists
        half = max(0.12, 0.5 * math.sqrt(case["n"] * SPACING ** 3 / 0.08))
        prm = dict(W.PHYS, box_half=(half, half, half), erosion=0)
        pos, vel = _pool(seed, case["n"], (half, half, half), torch.zeros(2, 2, device="cuda"))
        return prm, pos, vel
    half = _half(case["n"], "cube")
    pos, vel = _pool(seed, case["n"], half, torch.zeros(2, 2, device="cuda"))
    return dict(W.PHYS, box_half=half, erosion=0), pos, vel


def _requests(case, seed):
    rng = np.random.default_rng(seed)
    n = np.exp(rng.uniform(math.log(4096), math.log(case["n"]), case["requests"])).astype(int)
    side = rng.choice([64, 128, 256], case["requests"])
    steps = rng.integers(case["steps"] // 2, case["steps"] + 1, case["requests"])
    return [dict(seed=int(seed) * 1000 + i, particles=int(n[i]), terrain_side=int(side[i]), steps=int(steps[i]),
                 arrival_s=0.0) for i in range(case["requests"])]


# ---- the cases ---------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        inputs = _step_inputs(case, seed)
        total = sum(len(pos) for _, pos, _, _ in inputs)
        sysm = S.System(particle_capacity=sum((len(pos) + 511) // 512 * 512 for _, pos, _, _ in inputs),
                        terrain_capacity=sum((h.numel() + 511) // 512 * 512 for _, _, _, h in inputs),
                        tile=case["tile"], variant=case["variant"])
        st = dict(kind=kind, sys=sysm, steps=case["steps"], scenes=[], terrain_back=case["terrain_back"],
                  out=dict(pos=S.pinned_empty((total, 3)), vel=S.pinned_empty((total, 3)),
                           density=S.pinned_empty(total), sed=S.pinned_empty(total, np.int32)))
        at = 0
        for prm, pos, vel, h in inputs:
            sc = sysm.scene(S.default_params(**prm), capacity=len(pos), terrain=(h.shape[1], h.shape[0]))
            sc.set_terrain(h.cpu().numpy())
            sc.set_particles(pos.cpu().numpy(), vel.cpu().numpy())
            views = [st["out"][k][at:at + len(pos)] for k in ("pos", "vel", "density", "sed")]
            st["scenes"].append((sc, [C.c_void_p(v.ctypes.data) for v in views]))
            at += len(pos)
        return st
    if kind in ("frame", "record"):
        prm, pos, vel = _small_inputs(case, seed)
        flags = S.SPH_FLAG_RECORD | S.SPH_FLAG_ORDERED if kind == "record" else 0
        sysm = S.System(particle_capacity=len(pos))
        sc = sysm.scene(S.default_params(**prm, flags=flags), capacity=len(pos))
        sc.set_particles(pos.cpu().numpy(), vel.cpu().numpy())
        return dict(kind=kind, sys=sysm, scene=sc, pos=np.zeros((len(pos), 3), np.float32))
    if kind == "static":
        prm, pos, _ = _small_inputs(case, seed)
        return dict(kind=kind, prm=S.default_params(**prm), pos=pos.contiguous(),
                    density=torch.zeros(len(pos), device="cuda"), pressure=torch.zeros(len(pos), device="cuda"))
    if kind == "serve":
        server = S.Server(W.base_params(), variant=case["variant"], policy=1)
        return dict(kind=kind, server=server, requests=_requests(case, seed))
    if kind == "mesh":
        h = _heights(seed, case["tw"], case["td"], 0.3, False)
        fn = S.lib().sph_scene_terrain_mesh
        fn.restype, fn.argtypes = C.c_int, [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
        sysm = S.System(particle_capacity=512, terrain_capacity=h.numel())
        sc = sysm.scene(S.default_params(**dict(W.PHYS, box_half=(2.0, 0.5, 2.0))), terrain=(case["tw"], case["td"]))
        sc.set_terrain(h.cpu().numpy())
        return dict(kind=kind, sys=sysm, scene=sc, fn=fn, verts=np.zeros((h.numel(), 6), np.float32),
                    idx=np.zeros(6 * (case["tw"] - 1) * (case["td"] - 1), np.uint32))
    raise ValueError(kind)


def _ok(rc):
    if rc != 0:
        raise S.SphError(rc, S.lib().sph_last_error().decode())


def run(state):
    kind = state["kind"]
    if kind == "step":
        sysm = state["sys"]
        sysm.step(state["steps"])
        for sc, ptrs in state["scenes"]:
            _ok(S.lib().sph_scene_get_particles_async(sysm.h, sc.id, *ptrs))
        out = dict(state["out"])
        if state["terrain_back"]:
            out["heights"], out["delta"] = state["scenes"][0][0].get_terrain()
        return out
    if kind == "frame":
        state["sys"].step(1)
        return state["scene"].get_positions(state["pos"])
    if kind == "record":
        state["sys"].step(1)
        rec, nb = state["scene"].get_records()
        return dict(rec=rec, nb=nb)
    if kind == "static":
        pos = state["pos"]
        _ok(S.lib().sph_density_static(C.byref(state["prm"]), len(pos), C.c_void_p(pos.data_ptr()),
                                       C.c_void_p(state["density"].data_ptr()),
                                       C.c_void_p(state["pressure"].data_ptr()),
                                       C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return dict(density=state["density"], pressure=state["pressure"])
    if kind == "serve":
        res, _ = state["server"].run_trace(state["requests"])
        return dict(hash=np.array([r.state_hash for r in res], np.uint64).view(np.int64),
                    sediment=np.array([r.sediment_units for r in res], np.int64),
                    total=np.array([r.total_units for r in res], np.int64),
                    kinetic=np.array([r.kinetic for r in res], np.float64))
    _ok(state["fn"](state["sys"].h, state["scene"].id, C.c_void_p(state["verts"].ctypes.data),
                    C.c_void_p(state["idx"].ctypes.data)))
    return dict(verts=state["verts"], idx=state["idx"].view(np.int32))


# Neighbours within h of a particle, itself included, in these pools.
NEIGHBOURS = 55


def work(case):
    """Bytes: state read and written once a step (32 B each way per
    particle), what is read back, the terrain's heights and deltas.  Flops:
    the pair terms of the in-range neighbours, about 15 in the density pass
    and 50 in the force pass, and 100 a particle."""
    kind = case["kind"]
    if kind == "step":
        sc = _scenes(case)
        n, t = sum(a for a, _, _ in sc), sum(b * c for _, b, c in sc)
        return {"bytes": case["steps"] * (64 * n + 16 * t) + 32 * n + (12 * t if case["terrain_back"] else 0),
                "flops": case["steps"] * n * (65 * NEIGHBOURS + 100)}
    if kind == "frame":
        return {"bytes": 76 * case["n"], "flops": case["n"] * (65 * 20 + 100)}
    if kind == "record":
        return {"bytes": 176 * case["n"], "flops": case["n"] * (65 * 40 + 100)}
    if kind == "static":
        return {"bytes": 20 * case["n"], "flops": case["n"] * 15 * NEIGHBOURS}
    if kind == "serve":
        # log-uniform sizes and uniform step counts, at their means
        n = (case["n"] - 4096) / math.log(case["n"] / 4096)
        steps = case["requests"] * 0.75 * case["steps"]
        return {"bytes": steps * 64 * n, "flops": steps * n * (65 * 35 + 100)}
    v = case["tw"] * case["td"]
    return {"bytes": v * (4 + 24 + 24), "flops": 60 * v}


# ---- the step in 64 bits -------------------------------------------------------
PI = float(np.float32(3.141592))


def _f(v):
    return float(np.float32(v))


def _pairs(pos, h, lo, hi):
    """In-range pairs (i, j), self included, of particles [lo, hi) with all:
    cells of h in rows along x, three cells of nine rows around each."""
    mn = pos.min(0).values - 1e-9
    c = ((pos - mn) / (h * 1.000001)).long()
    dim = c.max(0).values + 3
    row = lambda y, z: (z * dim[1] + y) * dim[0]  # noqa: E731
    key = row(c[:, 1] + 1, c[:, 2] + 1) + c[:, 0] + 1
    order = torch.argsort(key)
    skey = key[order]
    for a in range(lo, hi, 1 << 19):
        i = torch.arange(a, min(hi, a + (1 << 19)), device=pos.device)
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                base = row(c[i, 1] + 1 + dy, c[i, 2] + 1 + dz) + c[i, 0] + 1
                st = torch.searchsorted(skey, base - 1)
                ln = torch.searchsorted(skey, base + 2) - st
                who = torch.repeat_interleave(i, ln)
                first = torch.repeat_interleave(st - (torch.cumsum(ln, 0) - ln), ln)
                j = order[first + torch.arange(len(who), device=pos.device)]
                near = ((pos[who] - pos[j]) ** 2).sum(1) <= h * h
                yield who[near], j[near]


def _density64(p, pos):
    h = p["h"]
    rho = torch.zeros(len(pos), dtype=torch.float64, device=pos.device)
    c6 = 315.0 / (64.0 * PI * h ** 9)
    for i, j in _pairs(pos, h, 0, len(pos)):
        s = ((pos[i] - pos[j]) ** 2).sum(1)
        rho.index_add_(0, i, p["mass"] * c6 * (h * h - s) ** 3)
    return rho, p["k"] * (rho - p["p0"])


def _surface(p, hgt, x, z):
    d, w = hgt.shape
    half = p["half"]
    sx, sz = (w - 1) / (2 * half[0]), (d - 1) / (2 * half[2])
    fx, fz = ((x + half[0]) * sx).clamp(0, w - 1), ((z + half[2]) * sz).clamp(0, d - 1)
    i, j = fx.long().clamp(max=w - 2), fz.long().clamp(max=d - 2)
    tx, tz = fx - i, fz - j
    f = hgt.reshape(-1)
    at = j * w + i
    h00, h10, h01, h11 = f[at], f[at + 1], f[at + w], f[at + w + 1]
    a0, a1 = h00 + tx * (h10 - h00), h01 + tx * (h11 - h01)
    dx = ((h10 - h00) + tz * ((h11 - h01) - (h10 - h00))) * sx
    dz = (a1 - a0) * sz
    nrm = torch.stack([-dx, torch.ones_like(dx), -dz], 1) / torch.sqrt(dx * dx + 1 + dz * dz)[:, None]
    near = (fz + 0.5).long().clamp(max=d - 1) * w + (fx + 0.5).long().clamp(max=w - 1)
    return -half[1] + a0 + tz * (a1 - a0), nrm, near


def _step64(p, pos, vel, sed, base, delta):
    """One step: (positions, velocities, density, sediment, the step's fields)."""
    h = p["h"]
    rho, P = _density64(p, pos)
    A, B = P / rho ** 2, p["mass"] / rho
    cs, cg = 45.0 / (PI * h ** 6), 945.0 / (32.0 * PI * h ** 9)
    fp, fv, nr = (torch.zeros_like(pos) for _ in range(3))
    lap = torch.zeros_like(rho)
    nb = torch.full_like(rho, -1.0)
    for i, j in _pairs(pos, h, 0, len(pos)):
        r = pos[i] - pos[j]
        s = (r * r).sum(1)
        lap.index_add_(0, i, B[j] * -cg * (h * h - s) * (3 * h * h - 7 * s))
        o = i != j
        i, j, r, s = i[o], j[o], r[o], s[o]
        ln = torch.sqrt(s)
        unit = torch.where((ln < 1e-4)[:, None], torch.full_like(r, 1 / math.sqrt(3)), r / ln.clamp(min=1e-30)[:, None])
        fp.index_add_(0, i, ((A[i] + A[j]) * p["mass"] * -cs * (h - ln) ** 2)[:, None] * unit)
        fv.index_add_(0, i, (B[j] * cs * (h - ln))[:, None] * (vel[j] - vel[i]))
        nr.index_add_(0, i, (B[j] * -cg * (h * h - s) ** 2)[:, None] * r)
        nb.index_reduce_(0, i, j.double(), "amax")
    g = torch.tensor(p["g"], dtype=torch.float64, device=pos.device)
    Fp, Fv, Fg = -fp * rho[:, None], fv * p["visc"], rho[:, None] * g
    Fs = -p["sigma"] * lap[:, None] * nr
    acc = (Fp + Fv + Fg + Fs) / rho[:, None]
    dt = p["dt"]
    v = vel + acc * dt
    x = pos + v * dt
    if base is not None:
        hgt = base + delta * p["unit"]
        y, nm, _ = _surface(p, hgt, x[:, 0], x[:, 2])
        low = x[:, 1] < y
        depth = y - x[:, 1]
        vn = (v * nm).sum(1)
        sp = v.norm(dim=1)
        f = 1 + torch.where(sp > 0, p["cr"] * depth / (dt * sp.clamp(min=1e-300)), torch.zeros_like(sp))
        v = torch.where((low & (vn < 0))[:, None], v - nm * (f * vn)[:, None], v)
        x[:, 1] = torch.where(low, y, x[:, 1])
    half = torch.tensor(p["half"], dtype=torch.float64, device=pos.device)
    out = ~(x.abs() < half).all(1)
    ax = (x.abs() / half).max(1).indices
    pick = torch.nn.functional.one_hot(ax, 3).double()
    sign = torch.sign((x * pick).sum(1))
    wall = torch.where(pick > 0, sign[:, None] * half, x)
    nm = -pick * sign[:, None]
    f = 1 + 0.5 * (x - wall).norm(dim=1) / (dt * v.norm(dim=1))
    v = torch.where(out[:, None], v - nm * (f * (v * nm).sum(1))[:, None], v)
    x = torch.where(out[:, None], wall, x)
    if base is not None and p["erosion"]:
        y, _, near = _surface(p, hgt, x[:, 0], x[:, 2])
        cap = (p["k_cap"] * v.norm(dim=1)).clamp(max=1.0) * 2.0 ** 30
        q = torch.where(sed < cap, p["k_pick"] * dt * (cap - sed), -p["k_dep"] * dt * (sed - cap))
        q = torch.where(x[:, 1] - y <= p["layer"], torch.minimum(torch.maximum(q, -sed), 2.0 ** 30 - sed), torch.zeros_like(q))
        sed = sed + q
        delta.reshape(-1).index_add_(0, near, -q)
    fields = (acc, P, Fp, Fv, Fg, Fs, nr, nb)
    return x, v, rho, sed, fields


def _consts(prm, tw=0, td=0):
    q = S.default_params(**prm)  # the parameter block as the caller holds it
    p = dict(h=_f(q.smoothing_radius), mass=_f(q.mass), k=_f(q.gas_stiffness), p0=_f(q.rest_density),
             visc=_f(q.viscosity), sigma=_f(q.surface_tension), dt=_f(q.dt), cr=_f(q.restitution),
             g=[_f(v) for v in q.gravity], half=[_f(v) for v in q.box_half], erosion=bool(q.erosion),
             k_cap=_f(q.k_capacity), k_pick=_f(q.k_pickup), k_dep=_f(q.k_deposit), layer=_f(q.erosion_layer))
    if tw:
        p["unit"] = p["mass"] / p["p0"] * 2.0 ** -30 / (4 * p["half"][0] * p["half"][2] / ((tw - 1) * (td - 1)))
    return p


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        got = []
        for prm, pos, vel, h in _step_inputs(case, seed):
            p = _consts(prm, h.shape[1], h.shape[0])
            x, v, base = pos.double(), vel.double(), h.double()
            sed, delta = torch.zeros(len(x), dtype=torch.float64, device="cuda"), torch.zeros_like(base)
            for _ in range(case["steps"]):
                x, v, rho, sed, _ = _step64(p, x, v, sed, base, delta)
            got.append((x, v, rho, base + delta * p["unit"]))
        out = dict(pos=torch.cat([a[0] for a in got]), vel=torch.cat([a[1] for a in got]),
                   density=torch.cat([a[2] for a in got]), sed=None)
        if case["terrain_back"]:
            out["heights"], out["delta"] = got[0][3], None
        return out
    if kind in ("frame", "record", "static"):
        prm, pos, vel = _small_inputs(case, seed)
        p = _consts(prm)
        x, v = pos.double(), vel.double()
        if kind == "static":
            rho, P = _density64(p, x)
            return dict(density=rho, pressure=P)
        x, v, rho, _, (acc, P, Fp, Fv, Fg, Fs, nr, nb) = _step64(p, x, v, torch.zeros_like(x[:, 0]), None, None)
        if kind == "frame":
            return x
        rec = torch.cat([x, v, acc, rho[:, None], P[:, None], Fp, Fv, Fg, Fs, nr, torch.zeros_like(rho)[:, None]], 1)
        return dict(rec=rec, nb=None)
    if kind == "mesh":
        h = _heights(seed, case["tw"], case["td"], 0.3, False).double()
        sx, sz = 4.0 / (case["tw"] - 1), 4.0 / (case["td"] - 1)
        # the sum of the four cross products of the edge vectors to the
        # neighbours that exist, normalised
        n = torch.zeros(*h.shape, 3, dtype=torch.float64, device="cuda")
        left, right, up, down = (torch.zeros_like(n) for _ in range(4))
        left[:, 1:, 0], left[:, 1:, 1] = sx, h[:, 1:] - h[:, :-1]
        right[:, :-1, 0], right[:, :-1, 1] = sx, h[:, 1:] - h[:, :-1]
        up[1:, :, 2], up[1:, :, 1] = sz, h[1:] - h[:-1]
        down[:-1, :, 2], down[:-1, :, 1] = sz, h[1:] - h[:-1]
        for a in (up, down):
            for b in (left, right):
                n += torch.linalg.cross(a, b)
        n /= n.norm(dim=2, keepdim=True)
        x = torch.arange(case["tw"], device="cuda").double() * sx - 2.0
        z = torch.arange(case["td"], device="cuda").double() * sz - 2.0
        v = torch.cat([torch.stack([x.expand_as(h), h - 0.5, z[:, None].expand_as(h)], 2), n], 2)
        return dict(verts=v.reshape(-1, 6), idx=None)
    return None
