"""Ray counts of a distant source around the 32 rays a warp takes and emits at
a time, with rays that pass beside the grid box: the tallies equal those of the
same rays materialised and cast one by one against every face, and of the
oracle where that is quick.  Tolerance: none."""
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
