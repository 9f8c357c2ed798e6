"""Calls whose faster route needs scratch memory, in a context whose budget has
no room for it: they take the route that needs none, with the same results."""
import numpy as np
import pytest

from form_factors_b200 import native, scenes

pytestmark = pytest.mark.gpu


def test_sinks_without_room_for_copies():
    faces = scenes.icosphere(1, 1.0, inward=False)
    n = len(faces)
    center, r = native.bounding_sphere(faces)
    source = native.DiscSource.make([0.3, -0.2, -1.0], center, 1.1 + 1.1 * r, 1.6 * r)
    front, power, mesh = np.full(n, 900, np.int32), np.ones(n, np.float32), (np.arange(n) % 5).astype(np.int32)
    zero = np.zeros(n, np.int32)
    one = np.ones(n, np.int32)

    def run(ctx):
        return (ctx.parallel_rays(source, 200000, seed=23),
                ctx.radiance_absorption(front, zero, power, power, mesh, 5, seed=3))

    free, tight = native.Context(0), native.Context(0)
    for c in (free, tight):
        c.scene_set(faces)
        c.grid_build()
    # every buffer but the copies: few rays (one copy), then the chunks of many
    tight.parallel_rays(source, 10, seed=1)
    tight.radiance_absorption(one, zero, power, power, mesh, 5, seed=3)
    out = np.zeros((n, n), np.uint32)
    tight.form_factor_counts(front, zero, 3, out=out)
    tight.set_budget(1)  # nothing may grow
    for a, b in zip(run(tight), run(free)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("factors", [False, True])
def test_host_output_without_room_for_pairs(factors):
    faces = scenes.icosphere(4, 1.0, inward=True)[:4400:2]
    n = len(faces)
    front, zero = np.full(n, 30, np.int32), np.zeros(n, np.int32)

    def run(ctx):
        return ctx.form_factors(front, zero, 9) if factors else ctx.form_factor_counts(front, zero, 9)

    tight = native.Context(0)
    tight.scene_set(faces)
    tight.grid_build(cells_per_face=16)
    tight.set_host_threads(0)  # dense
    want = run(tight)
    tight.set_budget(1)  # nothing may grow
    tight.set_host_threads(-1)
    assert np.array_equal(run(tight), want)
