"""Under a budget with no room for the faster routes' scratch the other routes are
the ones taken: the context's memory does not grow (it does without the budget),
and a host output crosses dense."""
import numpy as np
import pytest

from form_factors_b200 import native, scenes

pytestmark = pytest.mark.gpu


def test_sinks_keep_within_the_budget():
    faces = scenes.icosphere(1, 1.0, inward=False)
    n = len(faces)
    center, r = native.bounding_sphere(faces)
    source = native.DiscSource.make([0.3, -0.2, -1.0], center, 1.1 + 1.1 * r, 1.6 * r)
    many, zero, one = np.full(n, 900, np.int32), np.zeros(n, np.int32), np.ones(n, np.int32)
    power, mesh = np.ones(n, np.float32), (np.arange(n) % 5).astype(np.int32)
    results, grew = [], []
    for tight in (False, True):
        c = native.Context(0)
        c.scene_set(faces)
        c.grid_build()
        # every buffer but the copies of the counters
        c.parallel_rays(source, 10, seed=1)
        c.radiance_absorption(one, zero, power, power, mesh, 5, seed=3)
        c.form_factor_counts(many, zero, 3, out=np.zeros((n, n), np.uint32))
        before = c.device_bytes()
        if tight:
            c.set_budget(1)
        results.append((c.parallel_rays(source, 200000, seed=23),
                        c.radiance_absorption(many, zero, power, power, mesh, 5, seed=3)))
        grew.append(c.device_bytes() - before)
    assert grew[0] > 0 and grew[1] == 0
    for a, b in zip(*results):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("factors", [False, True])
def test_host_output_keeps_within_the_budget(factors):
    faces = scenes.icosphere(4, 1.0, inward=True)[:4400:2]
    n = len(faces)
    front, zero = np.full(n, 30, np.int32), np.zeros(n, np.int32)

    def run(c):
        return c.form_factors(front, zero, 9) if factors else c.form_factor_counts(front, zero, 9)

    free, tight = native.Context(0), native.Context(0)
    for c in (free, tight):
        c.scene_set(faces)
        c.grid_build(cells_per_face=16)
        c.set_host_threads(0)
        want = run(c)
        c.set_host_threads(-1)
    before = tight.device_bytes()
    tight.set_budget(1)
    assert np.array_equal(run(tight), want) and np.array_equal(run(free), want)
    assert tight.device_bytes() <= before
    assert free.stats().d2h_bytes < n * n
    if not factors:
        assert tight.stats().d2h_bytes == 4 * n * n
