"""Workloads of the lattice-Boltzmann library, as a user's program runs them.

Every case goes through the package's public entry points: the per-context
step (one cached or packet step with its output, or a window of resident steps
and a read of the state), the brick-world service (a tick and its packed
atlases), batched bricks (ticks, atlases and flows), the mesoscale grid (a
host-driven step, or a resident window), the wind grid's hydrodynamic
distribution alone, and the gradient of the differentiable brick.

`exact` restates each model in plain 64-bit torch; the brick world returns
whole numbers only and has no such value.
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import sys
import weakref
from pathlib import Path

import numpy as np
import torch
import torch.utils.checkpoint

ROOT = Path(__file__).resolve().parent.parent
PACKAGE = ROOT / "aerodynamics4mc-fabric_b200"

PERIODIC, BOUNCE_BACK, VELOCITY, CONVECTIVE = 1, 2, 4, 6
MAX_SPEED = float(np.float32(0.57735026919) * np.float32(0.60))


# ------------------------------------------------------------------ the cases
def listed() -> list[dict]:
    return [
        # The smallest call: one cached step of a small brick and its full
        # output, what a caller that follows one brick does every tick.
        {"name": "cached_step_16", "kind": "cached", "nx": 16, "ny": 16, "nz": 16, "variant": "fp32"},
        # One step with the caller's 11-channel packet (inputs change every
        # tick: the mask, the state and the sources come from the host).
        {"name": "packet_step_32", "kind": "packet", "nx": 32, "ny": 32, "nz": 32, "variant": "fp32"},
        # A ragged terrain brick in the library's default arithmetic (FP32,
        # reference order) with buoyancy, outflow and temperature transport:
        # a window of resident steps, then the state.
        {"name": "terrain_97x83x61_fp32", "kind": "terrain", "nx": 97, "ny": 83, "nz": 61, "variant": "fp32", "steps": 40},
        # The benchmark's 128^3 terrain brick in 16-bit fixed-point storage.
        {"name": "terrain_128_i16", "kind": "terrain", "nx": 128, "ny": 128, "nz": 128, "variant": "i16", "steps": 50},
        # The largest brick: a terrain of 6.3 million cells.
        {"name": "terrain_256x192x128_i16", "kind": "terrain", "nx": 256, "ny": 192, "nz": 128, "variant": "i16", "steps": 20},
        # The game's brick world as it ticks: eight 64^3 bricks, every tick
        # publishes their stride-4 packed atlases.
        {"name": "world_8x64", "kind": "world", "n": 64, "bx": 2, "by": 2, "bz": 2, "ticks": 1, "stride": 4},
        # The same service with many small bricks.
        {"name": "world_27x16", "kind": "world", "n": 16, "bx": 3, "by": 3, "bz": 3, "ticks": 1, "stride": 4},
        # Independent bricks of mixed sizes and precisions in one batch: 32
        # ticks with publishing, then every brick's atlas and flow.
        {"name": "batch_mixed_24", "kind": "batch", "small": 16, "mid": 6, "large": 2, "n_small": 32, "n_mid": 64, "n_large": 96,
         "ticks": 32},
        # The mesoscale grid driven from the host: 25-channel forcing in, state out.
        {"name": "meso_step_64x16x64", "kind": "meso_step", "nx": 64, "ny": 16, "nz": 64},
        # The mesoscale model resident on the device for a window of steps.
        {"name": "meso_window_128x24x128", "kind": "meso_window", "nx": 128, "ny": 24, "nz": 128, "steps": 30},
        # The wind field alone at the benchmark's 256 x 64 x 256, 16-bit storage.
        {"name": "hydro_256x64x256_i16", "kind": "hydro", "nx": 256, "ny": 64, "nz": 256, "storage": 2, "collision": 1, "steps": 60},
        # Loss and gradient through 200 steps of a 64^3 brick (forward and reverse).
        {"name": "adjoint_64", "kind": "adjoint", "n": 64, "steps": 200, "every": 20, "probes": 64},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["cached", "packet", "terrain", "terrain", "terrain", "world", "batch", "meso_step", "meso_window",
                       "hydro", "adjoint"])
    if kind in ("cached", "packet"):
        return {"kind": kind, "nx": rng.randint(8, 40), "ny": rng.randint(8, 40), "nz": rng.randint(8, 40),
                "variant": rng.choice(["fp32", "fp32", "fp32_fast", "i16", "fp16"])}
    if kind == "terrain":
        return {"kind": kind, "nx": _log(rng, 24, 256), "ny": _log(rng, 24, 192), "nz": _log(rng, 24, 128),
                "variant": rng.choice(["fp32", "fp32_fast", "i16", "i16", "fp16"]), "steps": rng.randint(6, 20)}
    if kind == "world":
        return {"kind": kind, "n": _log(rng, 12, 64), "bx": rng.randint(1, 2), "by": rng.randint(1, 2), "bz": rng.randint(1, 2),
                "ticks": rng.randint(1, 3), "stride": rng.choice([1, 2, 3, 4])}
    if kind == "batch":
        return {"kind": kind, "small": rng.randint(1, 16), "mid": rng.randint(1, 6), "large": rng.randint(0, 2),
                "n_small": rng.randint(15, 33), "n_mid": rng.randint(40, 66), "n_large": rng.randint(70, 96),
                "ticks": rng.randint(2, 24)}
    if kind == "meso_step":
        return {"kind": kind, "nx": _log(rng, 8, 96), "ny": rng.randint(2, 24), "nz": _log(rng, 8, 96)}
    if kind == "meso_window":
        return {"kind": kind, "nx": _log(rng, 12, 160), "ny": rng.randint(2, 32), "nz": _log(rng, 12, 160),
                "steps": rng.randint(4, 30)}
    if kind == "hydro":
        return {"kind": kind, "nx": _log(rng, 24, 256), "ny": _log(rng, 8, 64), "nz": _log(rng, 24, 256),
                "storage": rng.choice([0, 1, 2]), "collision": rng.choice([0, 1, 1]), "steps": rng.randint(6, 40)}
    return {"kind": kind, "n": rng.randint(16, 64), "steps": rng.randint(20, 120), "every": rng.choice([1, 7, 10, 20]),
            "probes": rng.randint(8, 64)}


# ------------------------------------------------------------------ inputs (from the seed alone)
def _rng(case: dict, seed: int) -> np.random.Generator:
    return np.random.default_rng([int(seed), sum(map(ord, case["kind"]))])


def _heightmap(n_x: int, n_y: int, octaves: int, amplitude: float, rng) -> np.ndarray:
    """Fractal value noise over the ground plane, scaled to [0, amplitude]."""
    h = torch.zeros(n_x, n_y, dtype=torch.float64)
    for k in range(octaves):
        m = 4 * 2 ** k + 1
        lattice = torch.from_numpy(rng.random((m, m)))[None, None]
        h += 0.5 ** k * torch.nn.functional.interpolate(lattice, size=(n_x, n_y), mode="bilinear", align_corners=True)[0, 0]
    h -= h.min()
    return (h * (amplitude / max(float(h.max()), 1e-9))).numpy()


def _porous(case: dict, seed: int) -> dict:
    """A porous brick: 5 % random solids over a solid floor, a noisy wind."""
    rng, dims = _rng(case, seed), (case["nx"], case["ny"], case["nz"])
    solid = (rng.random(dims) < 0.05).astype(np.uint8)
    solid[:, :, 0] = 1
    u0 = (0.05, 0.0, 0.0)
    u = [np.float32(u0[a]) + rng.uniform(-0.005, 0.005, dims).astype(np.float32) for a in range(3)]
    return {"dims": dims, "solid": solid, "u": u, "temperature": None, "u_ref": u0, "tau": 0.55, "c_sgs": 0.025, "beta": 0.0,
            "faces": [(PERIODIC, None)] * 4 + [(BOUNCE_BACK, None)] * 2}


def _terrain(case: dict, seed: int) -> dict:
    """Seeded terrain, inflow at x-, outflow at x+, far-field lid, a warm bubble
    over a lapse rate; buoyancy along z."""
    rng, dims = _rng(case, seed), (case["nx"], case["ny"], case["nz"])
    s = dims[2] / 128.0
    h = _heightmap(dims[0], dims[1], 4, 24.0 * s, rng)
    z = np.arange(dims[2])
    solid = (z[None, None, :] < h[:, :, None]).astype(np.uint8)
    solid[:, :, 0] = 1
    u_in = (0.08, 0.02, 0.0)
    u = [np.where(solid == 0, np.float32(v), np.float32(0)) for v in u_in]
    centre = (dims[0] * rng.uniform(0.4, 0.6), dims[1] * rng.uniform(0.4, 0.6), 20.0 * s)
    g = [np.exp(-((np.arange(n) - c) ** 2) / (2 * (8.0 * s) ** 2)) for n, c in zip(dims, centre)]
    temp = (0.01 * g[0][:, None, None] * g[1][None, :, None] * g[2][None, None, :] - 1e-3 * z[None, None, :]).astype(np.float32)
    far = (VELOCITY, u_in)
    return {"dims": dims, "solid": solid, "u": u, "temperature": temp, "u_ref": u_in, "tau": 0.55, "c_sgs": 0.1, "beta": 1e-4,
            "faces": [far, (CONVECTIVE, None), (PERIODIC, None), (PERIODIC, None), (BOUNCE_BACK, None), far]}


def _brick_inputs(case: dict, seed: int) -> dict:
    return _terrain(case, seed) if case["kind"] == "terrain" else _porous(case, seed)


def _reynolds(b: dict) -> float:
    speed = max([math.dist(b["u_ref"], (0, 0, 0))] + [math.dist(v, (0, 0, 0)) for _, v in b["faces"] if v])
    return speed / ((b["tau"] - 0.5) / 3.0)


def _batch_bricks(case: dict, seed: int) -> list[dict]:
    rng = _rng(case, seed)
    bricks = []
    for i, n in enumerate([case["n_small"]] * case["small"] + [case["n_mid"]] * case["mid"] + [case["n_large"]] * case["large"]):
        dims = (n, n, n)
        solid = (rng.random(dims, dtype=np.float32) < rng.uniform(0.0, 0.15)).astype(np.uint8)
        solid[:, :, 0] = 1
        u = [np.where(solid == 0, np.float32(v), np.float32(0)) + rng.uniform(-0.005, 0.005, dims).astype(np.float32) * (solid == 0)
             for v in (0.04, 0.01, 0.0)]
        bricks.append({"dims": dims, "solid": solid, "u": u, "tau": float(rng.uniform(0.51, 0.6)),
                       "force": rng.uniform(-1e-5, 1e-5, 3).astype(np.float32), "precision": i % 2,
                       "faces": [PERIODIC] * 4 + [BOUNCE_BACK] * 2})
    return bricks


CHANNELS = 25  # forcing channels of the mesoscale grid


def _meso_forcing(case: dict, seed: int) -> np.ndarray:
    """Terrain (y up), temperatures, roughness, humidity, winds, a convective
    cell and nested-grid corrections."""
    rng, (nx, ny, nz) = _rng(case, seed), (case["nx"], case["ny"], case["nz"])
    f = np.zeros((nx, ny, nz, CHANNELS), np.float32)
    h = _heightmap(nx, nz, 3, min(3.0, 0.5 * ny), rng)
    y = np.arange(ny)[None, :, None]
    f[..., 0] = h[:, None, :]
    f[..., 1] = 288.0
    f[..., 2] = 288.15 + rng.uniform(-2, 2, (nx, ny, nz))
    f[..., 3] = 289.65
    f[..., 4] = 290.0 + rng.uniform(-3, 3, (nx, 1, nz))
    f[..., 5] = rng.uniform(0.0, 2.0, (nx, 1, nz))
    f[..., 6] = 6.0
    f[..., 7] = 3.0
    f[..., 9] = rng.uniform(0.2, 0.8, (nx, ny, nz))
    f[..., 10] = rng.uniform(0.0, 0.5, (nx, ny, nz))
    f[..., 11] = rng.uniform(0.0, 0.05, (nx, ny, nz))
    f[..., 20] = rng.uniform(-0.3, 0.3, (nx, ny, nz))
    f[..., 21] = rng.uniform(-0.3, 0.3, (nx, ny, nz))
    f[..., 22] = rng.uniform(-0.2, 0.2, (nx, ny, nz))
    f[..., 24] = y < np.floor(h)[:, None, :]
    return f


HYDRO_OPTIONS = {"periodic_sides": 1, "free_slip_top": 1, "fixed_tau": 1, "tau_hydro": 0.52, "enable_sgs": 1, "smagorinsky_c": 0.1,
                 "body_force": (1e-6, 0.0, 0.0), "hydro_only": 1, "disable_edge_blend": 1}


def _hydro_forcing(case: dict, seed: int) -> np.ndarray:
    """A boundary layer over smooth terrain (y up), a log wind profile."""
    rng, (nx, ny, nz) = _rng(case, seed), (case["nx"], case["ny"], case["nz"])
    f = np.zeros((nx, ny, nz, CHANNELS), np.float32)
    h = _heightmap(nx, nz, 3, 12.0 * ny / 64.0, rng)
    y = np.arange(ny, dtype=np.float64)[None, :, None]
    f[..., 0] = h[:, None, :]
    f[..., 6] = (0.06 * np.log1p(y) / math.log(ny + 1.0)) * (64.0 / 5.0)
    f[..., 24] = y < h[:, None, :]
    return f


def _adjoint_inputs(case: dict, seed: int) -> dict:
    """A 5 % porous brick with a warm bubble; probe winds as if measured."""
    rng, n = _rng(case, seed), case["n"]
    solid = (rng.random((n, n, n)) < 0.05).astype(np.uint8)
    s, i = n / 64.0, np.arange(n)
    g = [np.exp(-((i - c) ** 2) / (2 * (6.0 * s) ** 2)) for c in (n / 2, n / 2, 16.0 * s)]
    temp = (0.01 * g[0][:, None, None] * g[1][None, :, None] * g[2][None, None, :] - 1e-3 * i[None, None, :]).astype(np.float32)
    phase = rng.uniform(0, 2 * math.pi, (3, 3))
    force = np.zeros((3, n, n, n), np.float32)
    for a in range(3):
        w = [np.cos(2 * math.pi * i / n * (1 + (a + k) % 3) + phase[a, k]) for k in range(3)]
        force[a] = 5e-6 * w[0][:, None, None] * w[1][None, :, None] * w[2][None, None, :]
    lo, hi = max(2, n // 8), n - max(2, n // 8)
    fluid = [(x * n + y) * n + z for x, y, z in rng.integers(lo, hi, (case["probes"] * 4, 3)) if solid[x, y, z] == 0]
    probes = np.array(rng.permutation(sorted(set(fluid)))[: case["probes"]], np.int32)
    targets = (np.array([0.05, 0.01, 0.0]) + rng.uniform(-0.01, 0.01, (len(probes), 3))).astype(np.float32)
    return {"solid": solid, "temperature": temp, "force": force, "inflow": (0.045, 0.012, 0.002), "probes": probes,
            "targets": targets}


# ------------------------------------------------------------------ the library
def _package():
    if "aero_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("aero_b200", PACKAGE / "__init__.py",
                                                      submodule_search_locations=[str(PACKAGE)])
        sys.modules["aero_b200"] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules["aero_b200"])
    return sys.modules["aero_b200"]


class _Runtime:
    """The process's one runtime: either contexts of the per-context API or the
    brick-world service owns it, as in a program that uses one of the two."""

    def __init__(self):
        self.owner, self.service, self.keys = None, None, 0

    def next_key(self) -> int:
        self.keys += 1
        return self.keys

    def library(self):
        lib = _package().load_library()
        lib.aero_lbm_b200_reset_tuning()
        lib.aero_lbm_set_realtime_solver_mode(0)
        lib.aero_lbm_benchmark_reset_config()
        return lib

    def contexts(self):
        lib = self.library()
        if self.owner != "contexts":
            if self.service is not None:
                self.service.release()
                self.service = None
            if not lib.aero_lbm_init_rect(32, 32, 32, 11, 4):
                raise RuntimeError(_package().last_error(lib))
            self.owner = "contexts"
        return lib

    def world_service(self):
        lib = self.library()
        if self.owner != "world":
            self.service = _package().BrickWorldService(lib)
            self.owner = "world"
        return self.service


_runtime = _Runtime()


def _pinned(*shape, dtype=torch.float32) -> np.ndarray:
    return torch.zeros(*shape, dtype=dtype, pin_memory=True).numpy()


class _State(dict):
    """What a program keeps between calls; `release` runs when it goes."""

    def on_release(self, fn, *args):
        weakref.finalize(self, fn, *args)
        return self

    __hash__ = object.__hash__


# solver mode, collision mode, 16-bit format
VARIANTS = {"fp32": (0, 0, 1), "fp32_fast": (0, 1, 1), "i16": (3, 1, 1), "fp16": (3, 1, 0)}


def _prepare_brick(case: dict, seed: int) -> _State:
    aero, lib, b = _package(), _runtime.contexts(), _brick_inputs(case, seed)
    mode, collision, fmt = VARIANTS[case["variant"]]
    lib.aero_lbm_set_realtime_solver_mode(mode)
    lib.aero_lbm_b200_set_fp16_format(fmt)
    lib.aero_lbm_b200_set_collision_mode(collision)
    buoyant = b["beta"] > 0
    lib.aero_lbm_b200_set_physics_overrides(b["c_sgs"], b["beta"], 2)
    ctx = aero.LbmContext(b["dims"], key=_runtime.next_key(), lib=lib, init=False)
    cfg = aero.default_config(lib)
    cfg.enabled = 1
    cfg.flags = (cfg.flags & ~aero.FLAG_DISABLE_SGS) | aero.FLAG_DISABLE_INTERNAL_THERMAL_SOURCE
    cfg.flags = cfg.flags & ~aero.FLAG_DISABLE_BUOYANCY if buoyant else cfg.flags | aero.FLAG_DISABLE_BUOYANCY
    cfg.reynolds_number = _reynolds(b)
    for a in range(3):
        cfg.initial_velocity[a] = b["u_ref"][a]
    for face, (kind, velocity) in zip(cfg.faces(), b["faces"]):
        face.hydrodynamic_kind = kind
        face.thermal_kind = 1
        for a in range(3):
            face.velocity[a] = velocity[a] if velocity else 0.0
    ctx.configure(cfg)
    if buoyant:
        ctx.set_temperature_state(b["temperature"])
    packet = aero.build_packet(b["solid"], *b["u"], temperature=b["temperature"])
    ctx.step(packet, output=False)
    state = _State(kind=case["kind"], ctx=ctx, lib=lib, steps=case.get("steps", 1), flow=_pinned(ctx.cells * 4))
    if buoyant:
        state["temperature"] = _pinned(ctx.cells)
    if case["kind"] == "packet":
        state["packet"] = torch.from_numpy(packet).pin_memory().numpy()
    return state.on_release(ctx.release)


def _checked(ok, lib):
    if not ok:
        raise RuntimeError(_package().last_error(lib))


def _run_brick(s: _State):
    aero, ctx, lib = _package(), s["ctx"], s["lib"]
    if s["kind"] == "cached":
        _checked(lib.aero_lbm_step_rect_cached(*ctx.dims, ctx.key, aero.fptr(s["flow"])), lib)
    elif s["kind"] == "packet":
        _checked(lib.aero_lbm_step_rect(aero.fptr(s["packet"]), *ctx.dims, ctx.key, aero.fptr(s["flow"])), lib)
    else:
        ctx.advance(s["steps"])
        _checked(lib.aero_lbm_get_flow_state_rect(*ctx.dims, ctx.key, aero.fptr(s["flow"])), lib)
        _checked(lib.aero_lbm_get_temperature_state_rect(*ctx.dims, ctx.key, aero.fptr(s["temperature"])), lib)
        return {"flow": s["flow"], "temperature": s["temperature"]}
    return s["flow"]


def _drop_world(aero, lib, service_key: int, world: int):
    lib.aero_lbm_simulation_submit_world_deltas(service_key, ctypes.byref(aero.AeroLbmWorldDelta(type=6, data0=world)), 1)


def _prepare_world(case: dict, seed: int) -> _State:
    """A world of equal bricks over one terrain (y up), with a few fans and heaters."""
    aero, svc, world, n = _package(), _runtime.world_service(), _runtime.next_key(), case["n"]
    rng, grid = _rng(case, seed), (case["bx"], case["by"], case["bz"])
    dims = tuple(n * b for b in grid)
    h = _heightmap(dims[0], dims[2], 4, 0.2 * dims[1], rng)
    solid = (np.arange(dims[1])[None, :, None] < np.maximum(h, 1.0)[:, None, :]).astype(np.uint8)
    flow = np.zeros(dims + (4,), np.float32)
    for a, v in enumerate((0.05, 0.0, 0.02)):
        flow[..., a] = np.where(solid == 0, np.float32(v) + rng.uniform(-0.005, 0.005, dims).astype(np.float32), 0)
    air = rng.uniform(-0.02, 0.02, dims).astype(np.float32)
    svc.ensure_world(world, n, dx=1.0, dt=0.05, solver_mode=1)
    coords = [(x, y, z) for x in range(grid[0]) for y in range(grid[1]) for z in range(grid[2])]
    svc.set_hints(world, coords)
    for k, c in enumerate(coords):
        cut = tuple(slice(c[a] * n, (c[a] + 1) * n) for a in range(3))
        kind, heat = np.zeros((n, n, n), np.uint8), np.zeros((n, n, n), np.float32)
        if k % 4 == 0:
            kind[n // 2, n // 2:n // 2 + 2, n // 2:n // 2 + 2] = 33  # fans blowing +x
        if k % 4 == 1:
            heat[n // 2, n // 2, n // 2:n // 2 + 2] = 400.0  # heaters, in watts
        svc.upload_static(world, c, solid[cut], surface_kind=kind, emitter=heat)
        svc.upload_dynamic(world, c, flow[cut], air[cut])
    svc.step(world, 1)
    res = (n + case["stride"] - 1) // case["stride"]
    atlases = _pinned(len(coords), res ** 3 * 4, dtype=torch.int16)
    state = _State(kind="world", svc=svc, world=world, coords=coords, ticks=case["ticks"], stride=case["stride"], atlases=atlases)
    return state.on_release(_drop_world, aero, svc.lib, svc.key, world)


def _run_world(s: _State):
    s["svc"].step(s["world"], s["ticks"])
    for c, out in zip(s["coords"], s["atlases"]):
        s["svc"].atlas(s["world"], c, s["stride"], out)
    return s["atlases"]


def _prepare_batch(case: dict, seed: int) -> _State:
    _runtime.contexts()
    batch = _package().BrickBatch()
    for b in _batch_bricks(case, seed):
        batch.add_brick(b["dims"], b["solid"], b["u"], b["tau"], b["force"], b["faces"], b["precision"])
    batch.finalize(stride=4, velocity_scale=20.0)
    batch.set_options(use_graph=True, publish=True)
    batch.tick(1)
    state = _State(kind="batch", batch=batch, ticks=case["ticks"])
    state["atlas"] = [_pinned(4 * math.prod(-(-d // 4) for d in dims), dtype=torch.int16) for dims in batch.dims]
    state["flow"] = [_pinned(math.prod(dims), 4) for dims in batch.dims]
    return state.on_release(batch.close)


def _run_batch(s: _State):
    b, lib = s["batch"], s["batch"].lib
    b.tick(s["ticks"])
    ok = True
    for i, (atlas, flow) in enumerate(zip(s["atlas"], s["flow"])):
        ok &= lib.aero_lbm_b200_batch_copy_atlas(b.handle, i, atlas.ctypes.data_as(ctypes.POINTER(ctypes.c_int16)), atlas.size)
        ok &= lib.aero_lbm_b200_batch_copy_flow(b.handle, i, _package().fptr(flow), flow.size)
    if not ok:
        raise RuntimeError(b.error())
    return {"atlas": s["atlas"], "flow": s["flow"]}


def _prepare_meso(case: dict, seed: int) -> _State:
    _runtime.contexts()
    aero, hydro = _package(), case["kind"] == "hydro"
    forcing = (_hydro_forcing if hydro else _meso_forcing)(case, seed).reshape(-1, CHANNELS)
    options = {**HYDRO_OPTIONS, "storage": case["storage"], "collision": case["collision"]} if hydro else None
    ctx = aero.MesoscaleContext((case["nx"], case["ny"], case["nz"]), options=options)
    state = _State(kind=case["kind"], ctx=ctx, steps=case.get("steps", 1), out=_pinned(ctx.cells, 6))
    ctx.step(forcing, state["out"])
    if case["kind"] == "meso_step":
        state["forcing"] = torch.from_numpy(forcing).pin_memory().numpy()
    return state.on_release(ctx.release)


def _run_meso(s: _State):
    ctx = s["ctx"]
    if s["kind"] == "meso_step":
        return ctx.step(s["forcing"], s["out"])
    ctx.advance(s["steps"])
    _checked(ctx.lib.aero_lbm_b200_mesoscale_read_state(ctx.key, _package().fptr(s["out"])), ctx.lib)
    return s["out"]


ADJOINT_MODEL = {"face_kind": (4, 4, 1, 1, 2, 4), "tau": 0.55, "smagorinsky_c": 0.1, "buoyancy_beta": 1e-4}


def _prepare_adjoint(case: dict, seed: int) -> _State:
    _runtime.contexts()
    p = _adjoint_inputs(case, seed)
    brick = _package().AdjointBrick(p["solid"], p["temperature"], steps=case["steps"], checkpoint_every=case["every"],
                                    **ADJOINT_MODEL)
    brick.set_probes(p["probes"], p["targets"])
    return _State(kind="adjoint", brick=brick, force=p["force"], inflow=p["inflow"]).on_release(brick.close)


def _run_adjoint(s: _State):
    loss, grad_force, grad_inflow = s["brick"].gradient(s["force"], s["inflow"])
    return {"loss": loss, "grad_force": grad_force, "grad_inflow": grad_inflow}


_PREPARE = {"cached": _prepare_brick, "packet": _prepare_brick, "terrain": _prepare_brick, "world": _prepare_world,
            "batch": _prepare_batch, "meso_step": _prepare_meso, "meso_window": _prepare_meso, "hydro": _prepare_meso,
            "adjoint": _prepare_adjoint}
_RUN = {"cached": _run_brick, "packet": _run_brick, "terrain": _run_brick, "world": _run_world, "batch": _run_batch,
        "meso_step": _run_meso, "meso_window": _run_meso, "hydro": _run_meso, "adjoint": _run_adjoint}


def prepare(case: dict, seed: int):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


# ------------------------------------------------------------------ work
def work(case: dict) -> dict:
    """Bytes and operations of one pass. A time step reads and writes every
    population once (plus the mask and the fields the model carries); the
    operations are those of the collision."""
    kind = case["kind"]
    if kind in ("cached", "packet", "terrain"):
        cells, steps = case["nx"] * case["ny"] * case["nz"], case.get("steps", 1)
        pops = 27 * 2 * (4 if case["variant"].startswith("fp32") else 2)
        per_step = pops + 1 + (32 if kind == "terrain" else 0)  # transport: state in and out, velocity in and out
        io = 16 + (4 if kind == "terrain" else 0) + (44 if kind == "packet" else 0)
        return {"bytes": cells * (steps * per_step + io), "flops": cells * steps * (1150.0 + (60 if kind == "terrain" else 0))}
    if kind == "world":
        bricks = case["bx"] * case["by"] * case["bz"]
        cells, samples = bricks * case["n"] ** 3, bricks * (-(-case["n"] // case["stride"])) ** 3
        # populations, mask and sources, the dynamic state (flow, air) out
        return {"bytes": cells * case["ticks"] * (216 + 10 + 20) + samples * 8, "flops": cells * case["ticks"] * 1250.0}
    if kind == "batch":
        sizes = [case["n_small"]] * case["small"] + [case["n_mid"]] * case["mid"] + [case["n_large"]] * case["large"]
        per = [n ** 3 * (27 * 2 * (2 if i % 2 else 4) + 1) for i, n in enumerate(sizes)]
        cells = sum(n ** 3 for n in sizes)
        return {"bytes": case["ticks"] * sum(per) + cells * 16 + sum((-(-n // 4)) ** 3 * 8 for n in sizes),
                "flops": case["ticks"] * cells * 1150.0}
    if kind in ("meso_step", "meso_window"):
        cells, steps = case["nx"] * case["ny"] * case["nz"], case.get("steps", 1)
        # two distributions and three temperature fields in and out, the forcing
        # channels the model reads
        return {"bytes": cells * (steps * (19 * 4 * 4 + 24 + 23 * 4) + 24), "flops": cells * steps * 900.0}
    if kind == "hydro":
        cells = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": cells * (case["steps"] * (19 * 2 * (2 if case["storage"] else 4) + 1) + 24),
                "flops": cells * case["steps"] * 420.0}
    cells = case["n"] ** 3
    # forward: populations in and out, temperature and force; reverse: state and
    # adjoint in, adjoint out, the force gradient accumulated
    return {"bytes": cells * (case["steps"] * (216 + 17 + 3 * 108 + 16) + 36), "flops": cells * case["steps"] * (1150.0 + 3600.0)}


# ------------------------------------------------------------------ 64-bit restatements
Q27 = [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)]
W27 = [(2 / 3 if x == 0 else 1 / 6) * (2 / 3 if y == 0 else 1 / 6) * (2 / 3 if z == 0 else 1 / 6) for x, y, z in Q27]
Q19 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, -1, 0),
       (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1)]
W19 = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12


def _f32(v) -> float:
    return float(np.float32(v))


def _device() -> torch.device:
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _d(a) -> torch.Tensor:
    return torch.as_tensor(np.ascontiguousarray(a), device=_device()).double()


def _feq(c, w, rho, u):
    cu = 3.0 * (c[0] * u[0] + c[1] * u[1] + c[2] * u[2])
    return w * rho * (1.0 + cu + 0.5 * cu * cu - 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]))


def _sums(line):
    """Orders 0, 1 and 2 over a direction's three populations."""
    return line[0] + line[1] + line[2], line[2] - line[0], line[2] + line[0]


def _back(m0, m1, m2, u):
    """Populations of a direction from its central moments about u."""
    r1 = m1 + u * m0
    r2 = m2 + 2.0 * u * m1 + u * u * m0
    return 0.5 * (r2 - r1), m0 - r2, 0.5 * (r1 + r2)


def _collide27(f, model: dict, force, temperature=None):
    """Cumulant collision with Smagorinsky relaxation and Guo forcing; the
    scheme's conservation fix-up vanishes in exact arithmetic. Returns the
    populations and the velocity used."""
    g = [[[f[(x * 3 + y) * 3 + z] for z in range(3)] for y in range(3)] for x in range(3)]
    sz = [[_sums(g[x][y]) for y in range(3)] for x in range(3)]
    sy0 = [_sums([sz[x][y][0] for y in range(3)]) for x in range(3)]
    sy1 = [_sums([sz[x][y][1] for y in range(3)]) for x in range(3)]
    r000, r100, r200 = _sums([sy0[x][0] for x in range(3)])
    r010, r110, _ = _sums([sy0[x][1] for x in range(3)])
    r020 = sum(sy0[x][2] for x in range(3))
    r001, r101, _ = _sums([sy1[x][0] for x in range(3)])
    r011 = sum(sy1[x][1] for x in range(3))
    r002 = sum(sz[x][y][2] for x in range(3) for y in range(3))
    rho = r000
    fx, fy, fz = force
    if temperature is not None:
        fz = fz + rho * (model["beta"] * temperature).clamp(-0.02, 0.02)
    u = [(r + 0.5 * b) / rho for r, b in ((r100, fx), (r010, fy), (r001, fz))]
    s2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    scale = torch.where(s2 > MAX_SPEED ** 2, MAX_SPEED / s2.clamp_min(1e-30).sqrt(), torch.ones_like(s2))
    ux, uy, uz = (v * scale for v in u)
    c200 = r200 - 2 * ux * r100 + ux * ux * rho
    c020 = r020 - 2 * uy * r010 + uy * uy * rho
    c002 = r002 - 2 * uz * r001 + uz * uz * rho
    c110 = r110 - ux * r010 - uy * r100 + ux * uy * rho
    c101 = r101 - ux * r001 - uz * r100 + ux * uz * rho
    c011 = r011 - uy * r001 - uz * r010 + uy * uz * rho
    eq = rho / 3.0
    n2 = (c200 - eq) ** 2 + (c020 - eq) ** 2 + (c002 - eq) ** 2 + 2.0 * (c110 ** 2 + c101 ** 2 + c011 ** 2)
    nu0, tau = model["nu0"], model["tau"]
    nut = (model["c_sgs"] ** 2 * n2.clamp_min(1e-60).sqrt() / (2.0 * rho * nu0).clamp_min(1e-6)).clamp_max(5.0 * nu0)
    lo = 0.5 + 3e-8
    tau_s = (0.5 + 3.0 * (nu0 + nut).clamp(1e-8, 0.15)).clamp(lo, 0.95)
    tau_n = (tau + (tau_s - tau) * _f32(0.30)).clamp(lo, 0.95)
    sd, so = (1.0 / tau_n).clamp(0.0, 1.95), (1.0 / tau_s).clamp(0.0, 1.95)
    a, b, c = (k + sd * (eq - k) for k in (c200, c020, c002))
    p, r, t = ((1.0 - so) * k for k in (c110, c101, c011))
    k220, k202, k022 = (a * b + 2 * p * p) / rho, (a * c + 2 * r * r) / rho, (b * c + 2 * t * t) / rho
    k211, k121, k112 = (a * t + 2 * p * r) / rho, (b * r + 2 * p * t) / rho, (c * p + 2 * r * t) / rho
    k222 = (a * b * c + 2 * p * p * c + 2 * r * r * b + 2 * t * t * a + 8 * p * r * t) / (rho * rho)
    zero = torch.zeros_like(rho)
    lines = {(0, 0): (rho, zero, a), (0, 1): (zero, r, zero), (0, 2): (c, zero, k202), (1, 0): (zero, p, zero),
             (1, 1): (t, zero, k211), (1, 2): (zero, k112, zero), (2, 0): (b, zero, k220), (2, 1): (zero, k121, zero),
             (2, 2): (k022, zero, k222)}
    gx = {bc: _back(*m, ux) for bc, m in lines.items()}
    pref = (1.0 - 0.5 * (1.0 / tau_s).clamp(0.0, 1.999)).clamp_min(0.0)
    uf = ux * fx + uy * fy + uz * fz
    out = [None] * 27
    for x in range(3):
        hy = [_back(gx[0, k][x], gx[1, k][x], gx[2, k][x], uy) for k in range(3)]
        for y in range(3):
            for z, v in enumerate(_back(hy[0][y], hy[1][y], hy[2][y], uz)):
                q = (x * 3 + y) * 3 + z
                e = Q27[q]
                cf = e[0] * fx + e[1] * fy + e[2] * fz
                cu = e[0] * ux + e[1] * uy + e[2] * uz
                out[q] = v + pref * W27[q] * (3.0 * (cf - uf) + 9.0 * cu * cf)
    return torch.stack(out), (ux, uy, uz)


def _plane(dims, axis: int, high: bool) -> torch.Tensor:
    m = torch.zeros(dims[axis], dtype=torch.bool, device=_device())
    m[-1 if high else 0] = True
    return m.view([-1 if k == axis else 1 for k in range(3)])


def _outflow(post, solid, faces, q: int):
    """Extrapolation from the two cells inward of the faces the pull leaves by."""
    first, second = [], []
    for k, n in enumerate(solid.shape):
        i = torch.arange(n, device=post.device)
        s = i - Q27[q][k]
        out = (s < 0) | (s >= n) if faces[2 * k][0] != PERIODIC else torch.zeros_like(s, dtype=torch.bool)
        step = torch.where(out, torch.full_like(i, Q27[q][k]), torch.zeros_like(i))
        first.append((i + step).clamp(0, n - 1))
        second.append((i + 2 * step).clamp(0, n - 1))
    at1, at2 = (torch.meshgrid(*v, indexing="ij") for v in (first, second))
    f1, f2 = post[q][at1], post[q][at2]
    f1 = torch.where(solid[at2], f1, f1 + _f32(0.15) * (f1 - f2))
    return torch.where(solid[at1], post[26 - q], torch.where(solid[at2], post[q][at1], f1))


def _pull27(post, solid, faces):
    out = []
    for q, c in enumerate(Q27):
        bounced = post[26 - q]
        v = torch.where(torch.roll(solid, c, (0, 1, 2)), bounced, torch.roll(post[q], c, (0, 1, 2)))
        for face in reversed(range(6)):
            kind, u = faces[face]
            if kind == PERIODIC or c[face // 2] != (-1 if face % 2 else 1):
                continue
            if kind == BOUNCE_BACK:
                w = bounced
            elif kind == VELOCITY:
                w = torch.as_tensor(_feq(c, W27[q], 1.0, u), dtype=torch.float64, device=post.device)
            else:
                w = _outflow(post, solid, faces, q)
            v = torch.where(_plane(solid.shape, face // 2, face % 2 == 1), w, v)
        out.append(v)
    return torch.stack(out)


def _macro27(f, solid):
    rho = f.sum(0).clamp(0.97, 1.03)
    u = [sum(c[a] * f[q] for q, c in enumerate(Q27) if c[a]) / rho for a in range(3)]
    o = torch.stack([*u, rho - 1.0], -1)
    return torch.where(solid[..., None], torch.zeros_like(o), o)


def _transport(t, solid, u):
    """Semi-Lagrangian advection by u, diffusion; walls and faces insulate."""
    n = t.shape
    i = [torch.arange(k, device=t.device).view([-1 if a == b else 1 for b in range(3)]) for a, k in enumerate(n)]

    def at(x, y, z):
        inside = (x >= 0) & (x < n[0]) & (y >= 0) & (y < n[1]) & (z >= 0) & (z < n[2])
        j = (x.clamp(0, n[0] - 1), y.clamp(0, n[1] - 1), z.clamp(0, n[2] - 1))
        return torch.where(inside & ~solid[j], t[j], t)

    pos = [i[a] - u[a] for a in range(3)]
    low = [p.floor() for p in pos]
    w = [p - k for p, k in zip(pos, low)]
    x, y, z = (k.long() for k in low)
    c = {(a, b, d): at(x + a, y + b, z + d) for a in (0, 1) for b in (0, 1) for d in (0, 1)}
    cx = {(b, d): c[0, b, d] + (c[1, b, d] - c[0, b, d]) * w[0] for b in (0, 1) for d in (0, 1)}
    cy = {d: cx[0, d] + (cx[1, d] - cx[0, d]) * w[1] for d in (0, 1)}
    adv = cy[0] + (cy[1] - cy[0]) * w[2]
    lap = sum(at(*[(i[a] + (d if a == k else 0)).expand(n) for a in range(3)]) for k in range(3) for d in (1, -1)) - 6.0 * t
    return torch.where(solid, torch.zeros_like(t), (adv + _f32(0.035) * lap).clamp(-1.0, 1.0))


def _exact_brick(case: dict, seed: int):
    b = _brick_inputs(case, seed)
    solid = _d(b["solid"]) != 0
    faces = [(k, None if v is None else tuple(_f32(x) for x in v)) for k, v in b["faces"]]
    speed = max(math.dist([_f32(x) for x in v], (0, 0, 0)) for v in [b["u_ref"]] + [v for _, v in b["faces"] if v])
    nu = _f32(_f32(speed) / _f32(_reynolds(b)))
    model = {"tau": _f32(0.5 + 3.0 * nu), "nu0": nu, "c_sgs": _f32(b["c_sgs"]), "beta": _f32(b["beta"])}
    u = tuple(_d(v) for v in b["u"])
    post = torch.stack([_feq(c, w, 1.0, u) for c, w in zip(Q27, W27)])
    u = tuple(torch.where(solid, torch.zeros_like(v), v) for v in u)
    t = None if b["temperature"] is None else _d(b["temperature"])
    zero = torch.zeros_like(u[0])
    rest = torch.tensor(W27, dtype=torch.float64, device=post.device).view(27, 1, 1, 1)
    for k in range(1 + case.get("steps", 1)):
        f = post if k == 0 else _pull27(post, solid, faces)
        if t is not None:
            t = _transport(t, solid, u)
        post, u = _collide27(f, model, (zero, zero, zero), t)
        post = torch.where(solid, rest, post)
        u = tuple(torch.where(solid, zero, v) for v in u)
    flow = _macro27(_pull27(post, solid, faces), solid).reshape(-1)
    return flow if t is None else {"flow": flow, "temperature": t.reshape(-1)}


def _exact_batch(case: dict, seed: int):
    flows = []
    for b in _batch_bricks(case, seed):
        solid, tau = _d(b["solid"]) != 0, _f32(b["tau"])
        model = {"tau": tau, "nu0": (tau - 0.5) / 3.0, "c_sgs": _f32(0.025), "beta": 0.0}
        faces = [(k, None) for k in b["faces"]]
        u = tuple(_d(v) for v in b["u"])
        post = torch.stack([_feq(c, w, 1.0, u) for c, w in zip(Q27, W27)])
        force = [torch.full_like(u[0], _f32(v)) for v in b["force"]]
        for k in range(1 + case["ticks"]):
            f = post if k == 0 else _pull27(post, solid, faces)
            post, _ = _collide27(f, model, force)
        flows.append(_macro27(_pull27(post, solid, faces), solid).reshape(-1, 4))
    return {"atlas": [None] * len(flows), "flow": flows}


def _opp19(q: int) -> int:
    return q if q == 0 else (q + 1 if q % 2 else q - 1)


def _odd_tau(even: float) -> float:
    return min(2.5, max(0.55, 0.5 + 0.25 / max(0.03, even - 0.5)))


class _Meso:
    """The mesoscale model: forcing-driven targets (or, with `hydro`, the
    distribution's own moments), two relaxation times, pull streaming."""

    def __init__(self, forcing: np.ndarray, hydro: bool):
        self.F, self.hydro = _d(forcing), hydro
        self.vs = _f32(64.0) / 5.0
        self.solid = self.F[..., 24] > 0.5
        self.wall = self.F[..., 4] + self.F[..., 23]
        nu = 1.5e-5 * 5.0 / 64.0 ** 2
        self.tau = HYDRO_OPTIONS["tau_hydro"] if hydro else min(2.5, max(0.58, 0.5 + 3.0 * nu))
        self.tau_t = min(2.5, max(0.58, 0.5 + nu / 0.71 / 0.25))
        F, vs = self.F, self.vs
        wind = [F[..., 6] + F[..., 20], F[..., 19] + F[..., 18], F[..., 7] + F[..., 21]]
        self.inflow = [(w / vs).clamp(-0.35, 0.35) for w in (wind[0] + F[..., 12] + F[..., 14], wind[1],
                                                              wind[2] + F[..., 13] + F[..., 15])]
        seed = [(torch.where(self.solid, torch.zeros_like(w), w) / vs).clamp(-0.35, 0.35) for w in wind]
        self.btemp = F[..., 2] + F[..., 22]
        self.ambient = torch.where(self.solid, self.wall, self.btemp)
        self.deep, self.surface = F[..., 3].clone(), self.wall.clone()
        self.f = torch.stack([_feq(c, w, 1.0, seed) for c, w in zip(Q19, W19)])
        self.g = torch.stack([self._geq(q, self.ambient, seed) for q in range(19)])

    @staticmethod
    def _geq(q, t, u):
        c = Q19[q]
        return W19[q] * t * (1.0 + 3.0 * (c[0] * u[0] + c[1] * u[1] + c[2] * u[2]))

    @staticmethod
    def _near(a, axis: int, d: int):
        """The neighbour along an axis, clamped at the edge."""
        i = (torch.arange(a.shape[axis], device=a.device) + d).clamp(0, a.shape[axis] - 1)
        return a.index_select(axis, i)

    def _moments(self):
        rho = self.f.sum(0)
        return rho, [sum(c[a] * self.f[q] for q, c in enumerate(Q19) if c[a]) / rho for a in range(3)], self.g.sum(0)

    def _targets(self, rho, u, amb):
        F, near = self.F, self._near
        lap = lambda a: near(a, 0, 1) + near(a, 0, -1) + near(a, 2, 1) + near(a, 2, -1) - 4.0 * a  # noqa: E731
        vlap = lambda a: near(a, 1, 1) + near(a, 1, -1) - 2.0 * a  # noqa: E731
        hum = (F[..., 9] + F[..., 11] + F[..., 17]).clamp(0.0, 1.0)
        sx = 0.5 * (near(F[..., 0], 0, 1) - near(F[..., 0], 0, -1))
        sz = 0.5 * (near(F[..., 0], 2, 1) - near(F[..., 0], 2, -1))
        ndeep = self.deep + 5.0 / 2400.0 * (F[..., 3] - self.deep) + 0.01 * vlap(self.deep)
        nsurf = (self.surface + 5.0 / 300.0 * (1.0 - 0.12 * hum) * (self.wall - self.surface) + 0.10 * (ndeep - self.surface)
                 + 0.04 * F[..., 10] + 0.08 * F[..., 16] + 0.05 * lap(self.surface) + 0.025 * vlap(self.surface))
        lx, ly, lz = self.inflow
        push = 0.0008 * (nsurf - amb)
        ny = rho.shape[1]
        near_ground = (1.0 - torch.arange(ny, device=rho.device, dtype=torch.float64) / max(1.0, ny - 1.0)).view(1, -1, 1)
        drag = (F[..., 5].clamp_min(0.0) * 0.02).clamp(0.0, 0.25)
        clamp = lambda v: v.clamp(-0.35, 0.35)  # noqa: E731
        goal = [clamp(lx - 0.005 * sx * lz + push * sx - drag * u[0]),
                clamp(ly + 0.0015 * (lx * sx + lz * sz) * near_ground + 0.0009 * (nsurf - amb) * near_ground - drag * u[1]),
                clamp(lz + 0.005 * sz * lx + push * sz - drag * u[2])]
        wr = 5.0 / 60.0
        v = [clamp((1.0 - wr) * a + wr * b) for a, b in zip(u, goal)]
        src = (5.0 / 600.0 * (self.btemp - amb) + (0.018 + 0.004 * hum) * (nsurf - amb) + 0.01 * (ndeep - amb)
               + 0.08 * F[..., 10] * (0.5 + 0.5 * hum) + 0.10 * F[..., 16] * (0.45 + 0.55 * hum) + 0.06 * F[..., 18]
               + 0.06 * F[..., 19] + 0.01 * lap(self.ambient) + 0.02 * vlap(self.ambient))
        pick = lambda a, b: torch.where(self.solid, a, b)  # noqa: E731
        return v, pick(self.wall, amb + src), pick(self.wall, nsurf), pick(F[..., 3], ndeep)

    def step(self):
        rho, u, amb = self._moments()
        one, zero = torch.ones_like(rho), torch.zeros_like(rho)
        if self.hydro:
            teq, nsurf, ndeep = zero, self.surface, self.deep
        else:
            u, teq, nsurf, ndeep = self._targets(rho, u, amb)
        rho = torch.where(self.solid, one, rho)
        u = [torch.where(self.solid, zero, v) for v in u]
        tu, om, force = u, torch.full_like(rho, 1.0 / self.tau), (0.0, 0.0, 0.0)
        if self.hydro:
            force = tuple(_f32(v) for v in HYDRO_OPTIONS["body_force"])
            tu = [torch.where(self.solid, zero, v + 0.5 * b / rho) for v, b in zip(u, force)]
            ne = [self.f[q] - _feq(Q19[q], W19[q], rho, tu) for q in range(19)]
            pi = {(a, b): sum(Q19[q][a] * Q19[q][b] * ne[q] for q in range(19) if Q19[q][a] * Q19[q][b])
                  for a in range(3) for b in range(a, 3)}
            n2 = sum((1.0 if a == b else 2.0) * v * v for (a, b), v in pi.items())
            nu0 = (self.tau - 0.5) / 3.0
            nut = (HYDRO_OPTIONS["smagorinsky_c"] ** 2 * n2.sqrt() / (2.0 * rho * nu0).clamp_min(1e-6)).clamp_max(5.0 * nu0)
            om = torch.where(self.solid, om, 1.0 / (0.5 + 3.0 * (nu0 + nut)))
        om_odd, gt_even, gt_odd = 1.0 / _odd_tau(self.tau), 1.0 / self.tau_t, 1.0 / _odd_tau(self.tau_t)
        uf = tu[0] * force[0] + tu[1] * force[1] + tu[2] * force[2]
        pf, pg = [], []
        for q, c in enumerate(Q19):
            o = _opp19(q)
            fe, feo = _feq(c, W19[q], rho, tu), _feq(Q19[o], W19[o], rho, tu)
            even, odd = 0.5 * (self.f[q] + self.f[o]), 0.5 * (self.f[q] - self.f[o])
            v = even - om * (even - 0.5 * (fe + feo)) + odd - om_odd * (odd - 0.5 * (fe - feo))
            if self.hydro:
                cf = c[0] * force[0] + c[1] * force[1] + c[2] * force[2]
                cu = c[0] * tu[0] + c[1] * tu[1] + c[2] * tu[2]
                v = v + torch.where(self.solid, zero, (1.0 - 0.5 * om) * W19[q] * (3.0 * (cf - uf) + 9.0 * cu * cf))
            pf.append(v)
            if not self.hydro:
                ge, geo = self._geq(q, teq, u), self._geq(o, teq, u)
                even, odd = 0.5 * (self.g[q] + self.g[o]), 0.5 * (self.g[q] - self.g[o])
                pg.append(even - gt_even * (even - 0.5 * (ge + geo)) + odd - gt_odd * (odd - 0.5 * (ge - geo)))
        self.deep, self.surface = ndeep, nsurf
        self._stream(pf, pg)

    def _stream(self, pf, pg):
        dims, dev = self.solid.shape, self.solid.device
        x, y, z = (torch.arange(n, device=dev).view([-1 if a == b else 1 for b in range(3)]) for a, n in enumerate(dims))
        edge = torch.minimum(torch.minimum(x, dims[0] - 1 - x), torch.minimum(z, dims[2] - 1 - z))
        sponge = torch.minimum(edge, dims[1] - 1 - y).expand(dims)
        alpha = torch.where(sponge <= 0, 1.0, torch.where(sponge < 2, 0.5, 0.0)).double()
        nof, nog, none = [], [], (0.0, 0.0, 0.0)
        for q, c in enumerate(Q19):
            o = _opp19(q)
            hit = torch.roll(self.solid, c, (0, 1, 2))
            ground = ((y - c[1]) < 0).expand(dims)
            out = ((x - c[0] < 0) | (x - c[0] >= dims[0]) | (z - c[2] < 0) | (z - c[2] >= dims[2])).expand(dims)
            lid = ((y - c[1]) >= dims[1]).expand(dims)
            fv = torch.roll(pf[q], c, (0, 1, 2))
            if self.hydro:  # periodic sides, a specular lid
                m = Q19.index((c[0], -c[1], c[2]))
                side = (c[0], 0, c[2])
                lid_hit = torch.roll(self.solid, side, (0, 1, 2))
                fv = torch.where(lid, torch.roll(pf[m], side, (0, 1, 2)), fv)
                fv = torch.where(ground | torch.where(lid, lid_hit, hit), pf[o], fv)
                nof.append(torch.where(self.solid, torch.full_like(fv, W19[q]), fv))
                continue
            fb, gb = _feq(c, W19[q], 1.0, self.inflow), self._geq(q, self.btemp, self.inflow)
            away = (out | lid) & ~ground
            bounced = ground | (hit & ~away)
            source = torch.where(ground, self.wall, torch.roll(self.wall, c, (0, 1, 2)))
            fv = torch.where(away, fb, fv)
            gv = torch.where(away, gb, torch.roll(pg[q], c, (0, 1, 2)))
            fv, gv = (1.0 - alpha) * fv + alpha * fb, (1.0 - alpha) * gv + alpha * gb
            fv, gv = torch.where(bounced, pf[o], fv), torch.where(bounced, W19[q] * source, gv)
            nof.append(torch.where(self.solid, torch.full_like(fv, W19[q]), fv))
            nog.append(torch.where(self.solid, W19[q] * self.wall, gv))
        self.f = torch.stack(nof)
        if not self.hydro:
            self.g = torch.stack(nog)
            self.ambient = torch.where(self.solid, self.wall, self.g.sum(0))

    def state(self):
        rho, u, amb = self._moments()
        zero, top = torch.zeros_like(rho), 0.35 * self.vs
        wind = [torch.where(self.solid, zero, (v * self.vs).clamp(-top, top)) for v in u]
        if self.hydro:
            return torch.stack([torch.where(self.solid, torch.ones_like(rho), rho), zero, zero, *wind], -1).reshape(-1, 6)
        return torch.stack([self.ambient, self.deep, self.surface, *wind], -1).reshape(-1, 6)


def _exact_meso(case: dict, seed: int):
    hydro = case["kind"] == "hydro"
    m = _Meso((_hydro_forcing if hydro else _meso_forcing)(case, seed), hydro)
    for _ in range(1 + case.get("steps", 1)):
        m.step()
    return m.state()


def _exact_adjoint(case: dict, seed: int):
    p, n = _adjoint_inputs(case, seed), case["n"]
    solid, t = _d(p["solid"]) != 0, _d(p["temperature"])
    tau = _f32(ADJOINT_MODEL["tau"])
    model = {"tau": tau, "nu0": (tau - 0.5) / 3.0, "c_sgs": _f32(ADJOINT_MODEL["smagorinsky_c"]),
             "beta": _f32(ADJOINT_MODEL["buoyancy_beta"])}
    kinds = ADJOINT_MODEL["face_kind"]
    force, inflow = _d(p["force"]).requires_grad_(), _d(np.float32(p["inflow"])).requires_grad_()
    rest = torch.tensor(W27, dtype=torch.float64, device=t.device).view(27, 1, 1, 1)

    def collide(f, force):
        post, _ = _collide27(f, model, (force[0], force[1], force[2]), t)
        return torch.where(solid, rest, post)

    def pull(post, inflow):
        out = []
        for q, c in enumerate(Q27):
            v = torch.where(torch.roll(solid, c, (0, 1, 2)), post[26 - q], torch.roll(post[q], c, (0, 1, 2)))
            for face in reversed(range(6)):
                if kinds[face] == PERIODIC or c[face // 2] != (-1 if face % 2 else 1):
                    continue
                w = post[26 - q] if kinds[face] == BOUNCE_BACK else _feq(c, W27[q], 1.0, inflow)
                v = torch.where(_plane(solid.shape, face // 2, face % 2 == 1), w, v)
            out.append(v)
        return torch.stack(out)

    def step(post, force, inflow):
        return collide(pull(post, inflow), force)

    ones = torch.ones_like(t)
    post = collide(torch.stack([_feq(c, w, 1.0, inflow) * ones for c, w in zip(Q27, W27)]), force)
    for _ in range(case["steps"] - 1):
        post = torch.utils.checkpoint.checkpoint(step, post, force, inflow, use_reentrant=False)
    f = pull(post, inflow).reshape(27, -1)[:, torch.as_tensor(p["probes"], device=t.device).long()]
    rho = f.sum(0).clamp(0.97, 1.03)
    u = torch.stack([sum(c[a] * f[q] for q, c in enumerate(Q27) if c[a]) / rho for a in range(3)], -1)
    loss = ((u - _d(p["targets"])) ** 2).sum()
    loss.backward()
    return {"loss": float(loss.detach()), "grad_force": force.grad, "grad_inflow": inflow.grad}


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "world":
        return None  # the service's atlases are whole numbers
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    return _exact_meso(case, seed) if kind.startswith("meso") or kind == "hydro" else _exact_brick(case, seed)
