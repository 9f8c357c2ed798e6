"""Grids whose test records are smaller than the L1 cache and larger (256 KB is
where the trace kernels stop caching them there): counts with and without
counters, in a matrix with and without the warp histogram, the cast, a distant
source and absorbed power, against the same rays cast against every face.
Tolerance: none (power: 1e-13 of the total, sums of doubles)."""
import numpy as np
import pytest

from form_factors_b200 import native, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [4, 8, 24, 48, 96])
@pytest.mark.parametrize("name", ["sphere", "clutter", "room"])
def test_every_sink(ctx, name, cells):
    faces = {"sphere": scenes.icosphere(2, 1.0, inward=True), "clutter": scenes.clutter(180, 0.08, seed=2, enclosure_cells=3),
             "room": scenes.enclosure(3, 22)}[name]  # 320, 288 and 3216 faces (2^22 entries and more: no histogram)
    n = len(faces)
    front, rear = np.full(n, 40, np.int32), np.full(n, 3, np.int32)
    ctx.scene_set(faces)
    ctx.grid_build(cells_per_face=cells)
    rays = ctx.emit(front, rear, 5)
    brute, points = ctx.cast(rays, brute=True)
    hit, pts = ctx.cast(rays)
    assert np.array_equal(hit, brute) and np.array_equal(pts.view(np.uint32), points.view(np.uint32))
    want = np.zeros((n, n), np.uint32)
    src = np.repeat(np.arange(n), front + rear)
    np.add.at(want, (src[hit >= 0], hit[hit >= 0]), 1)
    for on in (True, False):
        ctx.set_stats(on)
        assert np.array_equal(ctx.form_factor_counts(front, rear, 5), want)
        power = np.ones(n, np.float32)
        got = ctx.radiance_absorption(front, rear, power, power, np.arange(n, dtype=np.int32), n, seed=5)
        assert np.allclose(got, want.sum(0), rtol=0, atol=1e-13 * want.sum())
        center, r = native.bounding_sphere(faces)
        source = native.DiscSource.make([0.3, -0.2, -1.0], center, 1.1 + 1.1 * r, 1.1 * r)
        hits, _ = ctx.cast(ctx.emit_parallel(source, 5000, seed=7), want_points=False, brute=True)
        tally = ctx.parallel_rays(source, 5000, seed=7).sum(1)
        assert np.array_equal(tally, np.bincount(hits[hits >= 0], minlength=n))
    ctx.set_stats(True)
