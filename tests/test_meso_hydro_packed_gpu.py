"""The packed two-cell hydrodynamic step against the reference-order kernel on
grids where its pull can go wrong: a line of one pair, of a partial warp and of
a partial block, grids one or two cells high or wide, solid cells at the sides,
the ground and under the lid, and every option that changes the pull.

Tolerance: the two kernels differ in the order of FP32 sums only. A cell's
density or momentum is a sum of 19 populations whose absolute values add up to
about 1; at most 64 roundings of 2^-24 each touch a population per step, so
after 4 steps density and lattice wind (relative to sums of about 1) differ by
at most 4 * 64 * 2^-24 = 1.5e-5; wind is lattice wind times the velocity scale
dx / dt."""
from __future__ import annotations

import numpy as np
import pytest

import aero_b200
import oracle as O

pytestmark = pytest.mark.gpu

BOUND = 4 * 64 * 2.0**-24


@pytest.mark.parametrize("dims", [(1, 1, 2), (2, 2, 2), (3, 1, 4), (5, 4, 66), (4, 3, 258)])
@pytest.mark.parametrize("options", [{}, {"periodic_sides": 1}, {"free_slip_top": 1}, {"periodic_sides": 1, "free_slip_top": 1},
                                     {"disable_edge_blend": 1}, {"disable_edge_blend": 1, "periodic_sides": 1}])
def test_packed_step_equals_reference_order(gpu, dims, options):
    rng = np.random.default_rng(sum(dims))
    F = O.meso_forcing(dims, seed=sum(dims))
    F[rng.random(len(F)) < 0.15, 24] = 1.0
    base = {"hydro_only": 1, "fixed_tau": 1, "tau_hydro": 0.8, "body_force": (1e-4, 0.0, 2e-5), **options}
    got = {}
    for collision in (0, 1):
        ctx = aero_b200.MesoscaleContext(dims, dx_m=8.0, dt_s=2.0, options={**base, "collision": collision})
        try:
            ctx.step(F)
            ctx.advance(3)
            got[collision] = ctx.state().reshape(-1, 6)
        finally:
            ctx.release()
    d = np.abs(got[1].astype(np.float64) - got[0])
    assert np.isfinite(got[1]).all()
    assert d[:, 0].max() <= BOUND and d[:, 3:].max() <= BOUND * 4.0, (d[:, 0].max(), d[:, 3:].max())
