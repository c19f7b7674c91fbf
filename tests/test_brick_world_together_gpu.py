"""A tick steps a world's bricks together, up to 32 to a launch: worlds of 1, 2
and 33 bricks of ragged sizes give, bit for bit, the state of the same world
whose bricks step one by one (an identical static upload before each tick
marks every brick's forcing dirty, which takes that route)."""
from __future__ import annotations

import numpy as np
import pytest

import aero_b200

pytestmark = pytest.mark.gpu


def run(lib, n, coords, ticks, one_by_one):
    rng = np.random.default_rng(n * 100 + len(coords))
    svc = aero_b200.BrickWorldService(lib)
    try:
        svc.ensure_world(1, n)
        svc.set_hints(1, coords)
        static = {}
        for k, c in enumerate(coords):
            ob = (rng.random((n, n, n)) < 0.08).astype(np.uint8)
            ob[:, 0, :] = 1
            kind, heat = np.zeros((n, n, n), np.uint8), np.zeros((n, n, n), np.float32)
            kind[n // 2, n // 2, n // 2] = 32 + k % 6
            heat[n // 2, n // 2, n // 3] = 300.0
            static[c] = (ob, kind, heat)
            svc.upload_static(1, c, ob, surface_kind=kind, emitter=heat)
            flow = rng.uniform(-0.05, 0.05, (n, n, n, 4)).astype(np.float32)
            flow[..., 3] *= 0.05
            svc.upload_dynamic(1, c, flow, rng.uniform(-0.05, 0.05, (n, n, n)), rng.uniform(0, 0.02, (n, n, n)))
        out = []
        for _ in range(ticks):
            if one_by_one:
                for c in coords:
                    ob, kind, heat = static[c]
                    svc.upload_static(1, c, ob, surface_kind=kind, emitter=heat)
            svc.step(1, 1)
            out.append([np.concatenate([a.reshape(-1) for a in svc.dynamic(1, c)]) for c in coords]
                       + [svc.atlas(1, c, 3) for c in coords])
        return out
    finally:
        svc.release()


@pytest.mark.parametrize("n,shape", [(9, (1, 1, 1)), (13, (2, 1, 1)), (10, (11, 3, 1))])
def test_bricks_step_together_as_one_by_one(gpu, n, shape):
    coords = [(x, y, z) for x in range(shape[0]) for y in range(shape[1]) for z in range(shape[2])]
    a, b = run(gpu, n, coords, 5, False), run(gpu, n, coords, 5, True)
    for tick, (u, v) in enumerate(zip(a, b)):
        for k, (x, y) in enumerate(zip(u, v)):
            assert np.array_equal(x.view(np.uint8), y.view(np.uint8)), (tick, k)
    assert np.abs(a[-1][0]).max() > 1e-3
