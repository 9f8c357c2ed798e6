"""The launch shape of a context where none was chosen follows the scene's grid
(twelve references per face), and every shape, 0 among them, can be chosen."""
import numpy as np
import pytest

from form_factors_b200 import native, scenes

pytestmark = pytest.mark.gpu


def test_default_shape_follows_the_scene_until_one_is_set(oracle):
    c = native.Context(0)
    assert c.trace_shape() == 0
    c.set_stats(False)
    plates, clutter = scenes.parallel_plates(10, 1.0), scenes.clutter(400, 0.15, seed=3, enclosure_cells=3)
    seen = set()
    for faces, kw in ((plates, dict(dims=(4, 4, 4))), (clutter, dict(cells_per_face=256))):
        n = len(faces)
        c.scene_set(faces)
        c.grid_build(**kw)
        info = c.grid_info()
        want = 12 if info.n_refs < 12 * info.n_live_faces else 0
        seen.add(want)
        assert c.trace_shape() == want
        rays, zero = np.full(n, 50, np.int32), np.zeros(n, np.int32)
        assert np.array_equal(c.form_factor_counts(rays, zero, 3), oracle.form_factor_counts(faces, rays, zero, seed=3))
    assert seen == {0, 12}
    c.scene_set(plates)
    c.grid_build(dims=(4, 4, 4))
    for shape in (0, 12, 3):
        c.set_trace_shape(shape)
        assert c.trace_shape() == shape
