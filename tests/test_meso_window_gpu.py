"""A window of resident mesoscale steps (fused pull + collision with the
ambient pass between) leaves, bit for bit, the state of as many host-driven
steps with the same forcing, on grids one to a few cells wide, with solid
cells at the sides, the ground and under the lid, and with every option that
changes the pull."""
from __future__ import annotations

import numpy as np
import pytest

import aero_b200
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 3, 1), (8, 1, 9), (5, 4, 33), (17, 6, 8)])
@pytest.mark.parametrize("options", [None, {"periodic_sides": 1}, {"free_slip_top": 1}, {"periodic_sides": 1, "free_slip_top": 1},
                                     {"disable_edge_blend": 1}])
def test_window_equals_host_driven_steps(gpu, dims, options):
    rng = np.random.default_rng(sum(dims))
    F = O.meso_forcing(dims, seed=sum(dims))
    F[:, 10:19] = rng.uniform(-0.2, 0.2, (len(F), 9))
    F[:, 20:24] = rng.uniform(-0.3, 0.3, (len(F), 4))
    F[rng.random(len(F)) < 0.1, 24] = 1.0
    a, b = (aero_b200.MesoscaleContext(dims, options=options) for _ in range(2))
    try:
        a.step(F)
        b.step(F)
        for window in (1, 2, 5):
            a.advance(window)
            for _ in range(window):
                want = b.step(F)
            got = a.state()
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), window
        G = F[::-1].copy()  # the next call's forcing and mask differ
        assert np.array_equal(a.step(G).view(np.uint32), b.step(G).view(np.uint32))
        a.advance(3)
        for _ in range(3):
            want = b.step(G)
        assert np.array_equal(a.state().view(np.uint32), want.view(np.uint32))
    finally:
        a.release()
        b.release()
