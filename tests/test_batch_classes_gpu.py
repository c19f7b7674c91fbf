"""A batch steps its bricks class by class (storage, odd or even nz), one tile
per unit: whatever other bricks share the batch, whatever the launch shape, and
on sizes around a unit (one cell, one cell more than a tile's 128 or 256), each
brick's flow and atlas are, bit for bit, those of the brick alone."""
from __future__ import annotations

import numpy as np
import pytest

import aero_b200
import oracle as O

pytestmark = pytest.mark.gpu

DIMS = [(1, 1, 1), (1, 1, 2), (3, 3, 3), (1, 2, 128), (1, 2, 130), (1, 1, 129), (1, 1, 127), (6, 5, 8), (9, 7, 33), (20, 18, 16)]


def _brick(i: int, precision: int):
    rng = np.random.default_rng(10 * i + precision)
    dims = DIMS[i]
    u = [rng.uniform(-0.05, 0.05, dims).astype(np.float32) for _ in range(3)]
    faces = rng.choice([O.PERIODIC, O.BOUNCE_BACK], 3).repeat(2) if i % 3 else None
    return dims, (rng.random(dims) < 0.15).astype(np.uint8), u, 0.52 + 0.01 * i, (1e-5, 0, -2e-5), faces, precision


def _run(gpu, bricks, graph, tune):
    b = aero_b200.BrickBatch(gpu)
    for br in bricks:
        b.add_brick(*br)
    b.finalize(stride=2, velocity_scale=20.0)
    b.set_options(use_graph=graph, publish=True)
    if tune:  # the trial ticks are real ticks
        b.autotune(2)
        b.tick(60 - b.info()["ticks"])
    else:
        b.tick(60)
    assert b.info()["ticks"] == 60
    out = [(b.flow(i).tobytes(), b.atlas(i).tobytes()) for i in range(len(bricks))]
    b.close()
    return out


@pytest.mark.parametrize("precisions", [(0,), (1,), (0, 1)])
def test_brick_alone_and_in_company(gpu, precisions):
    bricks = [_brick(i, p) for i in range(len(DIMS)) for p in precisions]
    together = _run(gpu, bricks, True, False)
    assert _run(gpu, bricks, False, False) == together
    assert _run(gpu, bricks[::-1], True, False)[::-1] == together
    for k in range(0, len(bricks), 3):
        assert _run(gpu, [bricks[k]], True, False)[0] == together[k], DIMS[k // len(precisions)]


def test_launch_shapes_agree(gpu):
    bricks = [_brick(i, i % 2) for i in range(len(DIMS))]
    assert _run(gpu, bricks, True, True) == _run(gpu, bricks, True, False)
