"""The adjoint sweep's bookkeeping on the GPU: which states are kept,
recomputed or checkpointed must not change a bit of the gradient, on bricks
either side of the reverse launch's block-size line and with lengths around a
segment's; probes that name one cell add up in order (a probe named twice
doubles every adjoint value, exactly)."""
from __future__ import annotations

import numpy as np
import pytest

import aero_b200

pytestmark = pytest.mark.gpu


def problem(n, dims=None, seed=3):
    rng = np.random.default_rng(seed)
    dims = dims or (n, n, n)
    obstacle = (rng.random(dims) < 0.05).astype(np.uint8)
    temp = rng.uniform(-0.01, 0.01, dims).astype(np.float32)
    force = rng.uniform(-1e-5, 1e-5, (3,) + dims).astype(np.float32)
    fluid = np.flatnonzero(obstacle.reshape(-1) == 0)
    probes = rng.choice(fluid, 12, replace=False).astype(np.int32)
    targets = rng.uniform(-0.02, 0.05, (12, 3)).astype(np.float32)
    return obstacle, temp, force, probes, targets


def gradient(obstacle, temp, force, probes, targets, steps, every):
    b = aero_b200.AdjointBrick(obstacle, temp, face_kind=(4, 4, 1, 1, 2, 4), tau=0.55, smagorinsky_c=0.1,
                               buoyancy_beta=1e-4, steps=steps, checkpoint_every=every)
    try:
        b.set_probes(probes, targets)
        first = b.gradient(force, (0.05, 0.01, 0.0))
        again = b.gradient(force, (0.05, 0.01, 0.0))  # the buffers hold the last call's states now
        assert first[0] == again[0] and np.array_equal(first[1], again[1]) and np.array_equal(first[2], again[2])
        return first
    finally:
        b.close()


@pytest.mark.parametrize("dims,steps", [((9, 7, 5), 1), ((9, 7, 5), 2), ((13, 11, 10), 12), ((12, 10, 33), 13), ((54, 51, 53), 5)])
def test_checkpoint_interval_keeps_every_bit(gpu, dims, steps):
    p = problem(0, dims)
    want = gradient(*p, steps, 1)
    assert np.isfinite(want[0]) and np.all(np.isfinite(want[1])) and np.abs(want[1]).max() > 0
    for every in (2, 4, 5, 12, 40):
        got = gradient(*p, steps, every)
        assert got[0] == want[0] and np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2]), every


def test_probe_named_twice_doubles_the_gradient(gpu):
    obstacle, temp, force, probes, targets = problem(14)
    one = gradient(obstacle, temp, force, probes, targets, 6, 3)
    two = gradient(obstacle, temp, force, np.concatenate([probes, probes]), np.concatenate([targets, targets]), 6, 3)
    assert two[0] == pytest.approx(2 * one[0], rel=1e-14)
    assert np.array_equal(two[1], 2 * one[1]) and np.allclose(two[2], 2 * one[2], rtol=1e-13, atol=0)
