"""Which route a world's tick takes, by its kernel launches: 33 unchanged bricks
step in two groups of launches, with the three passes of the temperature update
in every other tick; after a static upload each brick steps on its own."""
from __future__ import annotations

import numpy as np
import pytest

import aero_b200

pytestmark = pytest.mark.gpu


def test_launches_of_a_tick(gpu):
    n, coords = 8, [(2 * x, 2 * y, 0) for x in range(11) for y in range(3)]  # no neighbours: no halo launches
    rng = np.random.default_rng(5)
    svc = aero_b200.BrickWorldService(gpu)
    try:
        svc.ensure_world(1, n)
        svc.set_hints(1, coords)
        obstacle = np.zeros((n, n, n), np.uint8)
        obstacle[:, 0, :] = 1
        for c in coords:
            svc.upload_static(1, c, obstacle)
            svc.upload_dynamic(1, c, rng.uniform(-0.05, 0.05, (n, n, n, 4)), rng.uniform(-0.05, 0.05, (n, n, n)))

        def tick():
            before = gpu.aero_lbm_b200_launch_count()
            svc.step(1, 1)
            return gpu.aero_lbm_b200_launch_count() - before

        for _ in range(2):
            tick()
        joint = [tick() for _ in range(4)]
        # inputs, step, output and at most the face pre-fill per group
        assert min(joint) in (2 * 3, 2 * 4), joint
        assert joint[0] == joint[2] and joint[1] == joint[3] and abs(joint[0] - joint[1]) == 2 * 3, joint
        for c in coords:
            svc.upload_static(1, c, obstacle)
        assert tick() >= 4 * len(coords)
    finally:
        svc.release()
