"""Launches on either side of each change of the chunk size (32, 64, 128 and 256
rays from 128 x 64, 128 and 256 rays per multiprocessor on): the rows of faces
scattered over the scene equal the oracle's, whose rays are keyed by face and index
(cpuFactorsCalculator/cpu_system.cpp:162-190).  Tolerance: none."""
import numpy as np
import pytest

from form_factors_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [64, 128, 256])
@pytest.mark.parametrize("beyond", [-1, 0])
def test_rows_equal_the_oracle(ctx, oracle, size, beyond):
    import torch
    total = size * 4 * 32 * torch.cuda.get_device_properties(0).multi_processor_count + beyond
    faces = scenes.clutter(180, 0.12, seed=7, enclosure_cells=3)
    n = len(faces)
    rng = np.random.default_rng(size)
    front = rng.multinomial(total * 2 // 3, np.full(n, 1.0 / n)).astype(np.int32)
    rear = rng.multinomial(total - int(front.sum()), np.full(n, 1.0 / n)).astype(np.int32)
    assert int(front.sum()) + int(rear.sum()) == total
    ctx.scene_set(faces)
    ctx.grid_build()
    got = ctx.form_factor_counts(front, rear, seed=9, epoch=1)
    pick = np.concatenate([[0, n - 1], rng.choice(np.arange(1, n - 1), 8, replace=False)])
    f, r = np.zeros_like(front), np.zeros_like(rear)
    f[pick], r[pick] = front[pick], rear[pick]
    want = oracle.form_factor_counts(faces, f, r, seed=9, epoch=1)
    assert np.array_equal(got[pick], want[pick])
