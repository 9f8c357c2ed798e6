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


@pytest.mark.parametrize("most", [0, 400000])
def test_one_face_with_most_rays(ctx, oracle, most):
    """Budgets far from even (one face emits nearly everything) and even ones take
    different loads of the test records, larger here than the L1 cache."""
    faces = scenes.clutter(600, 0.1, seed=5, enclosure_cells=7)
    n = len(faces)
    front, zero = np.full(n, 20, np.int32), np.zeros(n, np.int32)
    front[n // 2] += most
    ctx.scene_set(faces)
    ctx.grid_build()
    assert ctx.grid_info().n_refs * 64 > 256 << 10
    want = oracle.form_factor_counts(faces, front, zero, seed=3)
    assert np.array_equal(ctx.form_factor_counts(front, zero, seed=3), want)
    one = np.ones(n, np.float32)
    mesh = np.arange(n, dtype=np.int32)
    got = ctx.radiance_absorption(front, zero, one, one, mesh, n, seed=3)
    assert np.array_equal(np.rint(got).astype(np.int64), want.sum(0))  # whole numbers: one unit per ray
    ctx.batch_set([faces], cells_per_face=32)
    ctx.batch_prepare(front, zero, np.array([3], np.uint64))
    assert np.array_equal(_batch_counts(ctx, n), want)


def _batch_counts(ctx, n):
    import torch
    offs, words = ctx.batch_counts_layout()
    counts = torch.empty(words, dtype=torch.int32, device="cuda")
    ctx.batch_launch(counts, offs, advance_epoch=False)
    ctx.synchronize()
    return counts.cpu().numpy().view(np.uint32)[int(offs[0]):int(offs[0]) + n * n].reshape(n, n)
