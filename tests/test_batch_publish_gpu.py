"""The batch's publish launch takes blocks of 128 atlas records: bricks whose
record counts lie around that (one record, one block, one record more, ragged
sizes) publish the quantised values of their own flow, count for count."""
from __future__ import annotations

import numpy as np
import pytest

import aero_b200
from test_batch_gpu import quantize_signed, sampled

pytestmark = pytest.mark.gpu

DIMS = [(3, 3, 3), (32, 16, 16), (20, 21, 22), (1, 2, 512), (1, 2, 513), (5, 17, 31), (64, 32, 4)]


@pytest.mark.parametrize("stride", [1, 4, 7])
def test_publish_blocks_cover_every_record(gpu, stride):
    rng = np.random.default_rng(stride)
    b = aero_b200.BrickBatch(gpu)
    for i, dims in enumerate(DIMS):
        u = [rng.uniform(-0.05, 0.05, dims).astype(np.float32) for _ in range(3)]
        b.add_brick(dims, (rng.random(dims) < 0.1).astype(np.uint8), u, 0.55, (1e-5, 0, 0), None, i % 2)
    b.finalize(stride=stride, velocity_scale=20.0)
    for ticks in (1, 1, 5):
        b.tick(ticks)
        for i, dims in enumerate(DIMS):
            v = sampled(b.flow(i), dims, stride)
            want = np.stack([quantize_signed(v[:, k] * np.float32(20.0), 5.6) for k in range(3)] +
                            [quantize_signed(v[:, 3], 0.03)], axis=1)
            assert np.array_equal(b.atlas(i).reshape(-1, 4), want), (dims, ticks)
    b.close()
