"""Rays with one or two direction components far below the third (1e-30 to the
smallest float), whose distances to the planes of those axes overflow: casts equal
the brute-force definition (ray_caster/naive_cpu.cpp:65-97) bit for bit.
Tolerance: none."""
import numpy as np
import pytest

from form_factors_b200 import scenes

pytestmark = pytest.mark.gpu


def _rays(size, rng):
    out = []
    for axis in range(3):
        main, third = (axis + 1) % 3, (axis + 2) % 3
        for sign in (-1.0, 1.0):
            for p in range(30, 46):
                for kind in range(4):
                    o, e = np.zeros(3), np.zeros(3)
                    e[axis] = sign * 10.0 ** -p  # an origin of 0: the subtraction keeps it
                    if kind == 1:
                        e[third] = sign * 10.0 ** -p
                    else:
                        o[third] = e[third] = 0.4 * size * rng.uniform(-1, 1)
                    if kind == 2:
                        e[third] += 0.3 * size
                    o[main] = -2.0 * size if kind == 3 else 0.4 * size * rng.uniform(-1, 1)
                    e[main] = o[main] + (size if p % 2 else 1.0)
                    out.append(np.concatenate([o, e]))
    return np.array(out, np.float32)


@pytest.mark.parametrize("size", [0.02, 1.0, 30.0, 1e3])
def test_cast_equals_brute_force(ctx, oracle, size):
    # small faces are degenerate to the reference (dot(n, n) < 1e-8): only a box at 0.02
    faces = scenes.clutter(150, 0.1, seed=4, enclosure_cells=3) if size >= 1 else scenes.unit_box()
    faces = ((faces - np.float32(0.5)) * np.float32(size)).astype(np.float32)
    rays = _rays(size, np.random.default_rng(6))
    want, points = oracle.cast_naive(faces, rays)
    m = want >= 0
    assert m.mean() > 0.5
    ctx.scene_set(faces)
    for kw in (dict(), dict(dims=(1, 1, 1)), dict(dims=(32, 32, 32)), dict(dims=(256, 256, 256)),
               dict(dims=(2, 31, 256), skip_empty=False)):
        ctx.grid_build(**kw)
        hit, pts = ctx.cast(rays)
        assert np.array_equal(hit, want), "%s: %d of %d differ" % (kw, (hit != want).sum(), len(rays))
        assert np.array_equal(pts[m].view(np.uint32), points[m].view(np.uint32))
