"""The two forms of the reference-order in-place step. An explicit
set_cells_per_thread stands for every brick; without one, a brick whose
one-cell grid is a single wave takes the one-cell form and larger ones the
packed form. Both give the same bits through mask changes, cells reseeded
after a non-finite state and lines with a lone last cell, on bricks below and
above that line."""
from __future__ import annotations

from pathlib import Path

import numpy as np
import pytest

import aero_b200
import lbm_cases
import oracle as O
from test_d3q27_gpu import assert_bits
from test_inplace_gpu import local_faces_case

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).resolve().parent / "golden"
SMALL, LARGE = (20, 12, 13), (60, 44, 35)  # line-padded cells 7,680 and 168,960; one wave: 75,776


def form(gpu, cpt):
    gpu.aero_lbm_b200_reset_tuning()  # no explicit form
    if cpt:
        assert gpu.aero_lbm_b200_set_cells_per_thread(cpt) == 1


def context(gpu, dims, cpt, key):
    """Faces of every local kind, x and z not periodic, one call done."""
    rng = np.random.default_rng(sum(dims))
    obst = (rng.random(dims) < 0.07).astype(np.uint8)
    u = [rng.uniform(-0.01, 0.01, dims).astype(np.float32) for _ in range(3)]
    form(gpu, cpt)
    ctx = aero_b200.LbmContext(dims, key=key, lib=gpu)
    ctx.configure(lbm_cases.product_config(gpu, local_faces_case()[3]))
    ctx.step(O.packet_from(obst, *u), output=False)
    return ctx, obst, u, rng


@pytest.mark.parametrize("dims", [SMALL, LARGE])
@pytest.mark.parametrize("cpt", [None, 1, 2])
def test_form_that_runs(gpu, dims, cpt):
    import torch
    from torch.profiler import ProfilerActivity, profile

    ctx = context(gpu, dims, cpt, key=300)[0]
    torch.cuda.init()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        ctx.advance(2)
        torch.cuda.synchronize()
    names = {e.key for e in p.key_averages()}
    packed = any("step_ip2_kernel" in k for k in names)
    single = any("step_ip_kernel" in k for k in names)
    assert packed != single, names
    assert packed == (cpt == 2 or (cpt is None and dims == LARGE)), (cpt, names)


@pytest.mark.parametrize("dims", [SMALL, LARGE, (40, 48, 34)])
def test_forms_give_the_same_bits(gpu, dims):
    outs = []
    for cpt in (1, 2, None):
        ctx, obst, u, rng = context(gpu, dims, cpt, key=301)
        ctx.advance(3)
        # a non-finite state at a few cells, both lanes of a pair among them
        force = np.zeros((3,) + dims, np.float32)
        force[0, 3, 4, 5] = force[1, 5, 6, 8] = force[2, 5, 6, 9] = force[0, 7, 8, dims[2] - 1] = np.inf
        ctx.set_force_field(*force)
        ctx.advance(1)
        ctx.set_force_field(*np.zeros_like(force))
        ctx.advance(3)
        flip = rng.random(dims)
        obst = np.where(obst == 1, flip < 0.5, flip < 0.04).astype(np.uint8)
        ctx.step(O.packet_from(obst, *u), output=False)
        ctx.advance(2)
        outs.append(ctx.step(None, output=True))
        ctx.release()
    assert np.isfinite(outs[0]).all() and np.abs(outs[0][:, :3]).max() > 1e-3
    assert_bits(outs[1], outs[0])
    assert_bits(outs[2], outs[0])


def test_packed_form_golden(gpu):
    g = np.load(GOLDEN / "c1_32_1000.npz")
    n = int(g["n"])
    obst, u = O.c1_inputs(seed=int(g["seed"]), n=n)
    form(gpu, 2)
    out, _ = lbm_cases.run_product(gpu, (n, n, n), O.c1_config(), O.packet_from(obst, *u), int(g["steps"]), streaming_mode=0)
    assert_bits(out, g["out"])
