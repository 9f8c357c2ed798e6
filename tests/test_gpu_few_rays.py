"""Faces with few rays: a warp fills its queue of 32 rays from many chunks, each
published to its lanes through shared memory.  Counts of every launch shape, with
and without counters, in a small matrix (warp histogram) and a large one, equal
the oracle's (cpuFactorsCalculator/cpu_system.cpp:162-190).  Tolerance: none."""
import numpy as np
import pytest

from form_factors_b200 import native, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("most", [1, 3, 31, 45])
@pytest.mark.parametrize("large", [False, True])
def test_many_chunks_per_fill(ctx, oracle, most, large):
    faces = scenes.icosphere(3, 1.0, inward=True) if large else scenes.clutter(180, 0.1, seed=5, enclosure_cells=3)
    n = len(faces)
    rng = np.random.default_rng(most)
    front, rear = rng.integers(0, most + 1, n).astype(np.int32), rng.integers(0, 2, n).astype(np.int32)
    want = oracle.form_factor_counts(faces, front, rear, seed=3, epoch=2)
    ctx.scene_set(faces)
    ctx.grid_build()
    assert np.array_equal(ctx.form_factor_counts(front, rear, seed=3, epoch=2), want)
    ctx.set_stats(False)
    for shape in range(len(native.trace_shapes())):
        ctx.set_trace_shape(shape)
        got = ctx.form_factor_counts(front, rear, seed=3, epoch=2)
        assert np.array_equal(got, want), "shape %d: %d entries differ" % (shape, (got != want).sum())
    ctx.set_trace_shape(0)
    ctx.set_stats(True)
