"""Sinks with few counters: a distant source's tallies and absorbed power.

Ray counts of a distant source around the 32 rays a warp takes and emits at
a time, with rays that pass beside the grid box: the tallies equal those of the
same rays materialised and cast one by one against every face, and of the
oracle where that is quick.  Tolerance: none.

Absorbed power by few and many meshes, whose counters are kept in many copies
or in one: sums over meshes of the power absorbed face by face.  Both are sums
of the same 64-bit integers; turning 80 of them into doubles and adding those
loses at most 80 * 2^-53 of the total, and the tolerance is 1e-13."""
import numpy as np
import pytest

from form_factors_b200 import native, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 31, 32, 33, 63, 64, 65, 255, 257, 4736, 151553, 1212417])
def test_tallies_at_batch_edges(ctx, oracle, n):
    faces = scenes.icosphere(1, 1.0, inward=False)
    center, r = native.bounding_sphere(faces)
    src = ([0.3, -0.2, -1.0], center, 1.1 + 1.1 * r, 1.6 * r)  # a disc wider than the scene
    ctx.scene_set(faces)
    ctx.grid_build()
    source = native.DiscSource.make(*src)
    got = ctx.parallel_rays(source, n, seed=23, epoch=1)
    hit, _ = ctx.cast(ctx.emit_parallel(source, n, seed=23, epoch=1), want_points=False, brute=True)
    assert np.array_equal(got.sum(1), np.bincount(hit[hit >= 0], minlength=len(faces)))
    if n <= 151553:
        assert np.array_equal(got, oracle.parallel_rays(faces, oracle.disc_source(*src), n, seed=23, epoch=1))


@pytest.mark.parametrize("meshes", [1, 2, 15, 16, 17, 33, 79])
@pytest.mark.parametrize("rays", [1, 40, 3000])
def test_absorption_in_copies(ctx, meshes, rays):
    faces = scenes.icosphere(1, 1.0, inward=True)
    n = len(faces)
    front, rear = np.full(n, rays, np.int32), np.zeros(n, np.int32)
    power = np.random.default_rng(meshes).random(n).astype(np.float32)
    ctx.scene_set(faces)
    ctx.grid_build()
    each = ctx.radiance_absorption(front, rear, power, power, np.arange(n, dtype=np.int32), n, seed=3)
    mesh = (np.arange(n) % meshes).astype(np.int32)
    got = ctx.radiance_absorption(front, rear, power, power, mesh, meshes, seed=3)
    want = np.bincount(mesh, weights=each, minlength=meshes)
    assert each.sum() > 0
    assert np.allclose(got, want, rtol=0, atol=1e-13 * each.sum())
