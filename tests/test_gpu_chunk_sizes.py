"""A launch's rays go to its warps in chunks of 32 to 256 rays, by the number of
rays in the launch; the counts are integer sums, so they do not depend on the
chunks.  A launch on either side of each change of the chunk size is compared
with the same matrix traced in row blocks, whose smaller launches take smaller
chunks, and with single faces' rows from the oracle (their rays are keyed by
face and index, cpuFactorsCalculator/cpu_system.cpp:162-190).  Tolerance: none."""
import numpy as np
import pytest

from form_factors_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thousands", [1, 605, 607, 1211, 1214, 2424, 2426, 4848, 4852])
def test_counts_do_not_depend_on_the_chunks(ctx, oracle, thousands):
    faces = scenes.clutter(180, 0.12, seed=7, enclosure_cells=3)
    n = len(faces)
    total = thousands * 1000
    rng = np.random.default_rng(thousands)
    front = rng.multinomial(total * 2 // 3, np.full(n, 1.0 / n)).astype(np.int32)
    rear = rng.multinomial(total - front.sum(), np.full(n, 1.0 / n)).astype(np.int32)
    front[5], rear[5], front[6] = 0, 0, 1
    ctx.scene_set(faces)
    ctx.grid_build()
    got = ctx.form_factor_counts(front, rear, seed=9, epoch=1)
    rows = [ctx.form_factor_counts_rows(front, rear, 9, a, b, epoch=1)
            for a, b in ((0, 1), (1, n // 7), (n // 7, n // 2), (n // 2, n))]
    assert np.array_equal(got, np.concatenate(rows))
    assert not got[5].any() and got[6].sum() <= 1 + rear[6]
    f, r = np.zeros_like(front), np.zeros_like(rear)
    for face in (6, n - 1):
        f[face], r[face] = min(front[face], 500), 0
    want = oracle.form_factor_counts(faces, f, r, seed=9, epoch=1)
    assert np.array_equal(ctx.form_factor_counts(f, r, seed=9, epoch=1), want)
