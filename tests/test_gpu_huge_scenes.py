"""Scenes with a face so large that the reference's own arithmetic overflows on it
(and never reports a hit there), up to an extent beyond the largest float: the other
faces are found as by the brute-force definition (ray_caster/naive_cpu.cpp:65-97).
Tolerance: none."""
import numpy as np
import pytest

from form_factors_b200 import scenes
import rays as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [1e6, 1e12, 1e19, 1e25, 1e30, 1e36, 1.6e38, 1.7e38, 2.5e38, 3.4e38])
def test_cast_beside_a_huge_face(ctx, oracle, far):
    faces = scenes.clutter(60, 0.2, seed=4, enclosure_cells=2)
    f = far
    big = np.array([[-f, f, -f, f, f, -f, 0, f, f], [f, -f, -f, f, f, 0, f, 0, f]], np.float32)
    rays = R.mixed_rays(np.random.default_rng(3), faces, 900)
    faces = np.concatenate([big[:1], faces, big[1:]]).astype(np.float32)
    want, points = oracle.cast_naive(faces, rays)
    m = want >= 0
    assert m.mean() > 0.3
    ctx.scene_set(faces)
    for kw in (dict(), dict(dims=(8, 8, 8)), dict(dims=(3, 200, 5), skip_empty=False)):
        ctx.grid_build(**kw)
        hit, pts = ctx.cast(rays)
        assert np.array_equal(hit, want), "%g %s: %d of %d differ" % (far, kw, (hit != want).sum(), len(rays))
        assert np.array_equal(pts[m].view(np.uint32), points[m].view(np.uint32))
