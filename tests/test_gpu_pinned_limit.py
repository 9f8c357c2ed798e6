"""Host outputs on a host that cannot page-lock memory for them: outputs below
64 MB, which need none, are written all the same; a larger one reports the failed
allocation, and that error is gone for the calls after it.  Tolerance: none."""
import numpy as np
import pytest

from form_factors_b200 import native, scenes

pytestmark = pytest.mark.gpu


def _limit(ctx, n_bytes):
    import ctypes
    fn = native.load().ffb_test_pinned_limit
    fn.argtypes, fn.restype = [ctypes.c_void_p, ctypes.c_ulonglong], None
    fn(ctx._h, n_bytes)


def test_outputs_without_pinned_memory():
    faces = np.concatenate([scenes.icosphere(4, 1.0, inward=True)] * 2)[:4400]
    n, small = len(faces), 2300
    rays = np.full(n, 60, np.int32)
    zero = np.zeros(n, np.int32)

    def solve(c, n, factors):
        return (c.form_factors if factors else c.form_factor_counts)(rays[:n], zero[:n], 9)

    free, tight = native.Context(0), native.Context(0)
    _limit(tight, 1)
    for c in (free, tight):
        c.scene_set(faces[:small])
        c.grid_build(cells_per_face=16)
    for factors in (False, True):
        assert np.array_equal(solve(tight, small, factors), solve(free, small, factors))
    for c in (free, tight):
        c.scene_set(faces)
        c.grid_build(cells_per_face=16)
    assert n * n * 4 >= 64 << 20
    want = solve(free, n, False)
    with pytest.raises(native.FFBError, match="memory"):
        solve(tight, n, False)
    _limit(tight, 0)
    assert np.array_equal(solve(tight, n, False), want)
    _limit(tight, 1 << 30)
    assert np.array_equal(solve(tight, n, True), solve(free, n, True))


def test_factors_without_room_for_dense_blocks():
    """A budget that holds the pairs of the row blocks but not the block that a
    dense one would be normalised in: nothing is launched before that is known."""
    n = 2200
    faces = scenes.icosphere(4, 1.0, inward=True)[:2 * n:2]
    front, zero = np.full(n, 540, np.int32), np.zeros(n, np.int32)
    front[0] = 70000  # pairs of two words: half the matrix
    free, tight = native.Context(0), native.Context(0)
    for c in (free, tight):
        c.scene_set(faces)
        c.grid_build(cells_per_face=16)
        c.form_factor_counts(front, zero, 1)
    before, matrix = tight.device_bytes(), 4 * n * n
    tight.set_budget(before + int(0.58 * matrix))
    assert np.array_equal(tight.form_factors(front, zero, 9), free.form_factors(front, zero, 9))
    assert tight.device_bytes() - before > 0.4 * matrix  # two dense matrices for one and the pairs
    assert np.array_equal(tight.form_factors(front, zero, 10), free.form_factors(front, zero, 10))


@pytest.mark.parametrize("rays", [30, 990, 1024])
def test_small_outputs_lock_no_memory(rays):
    """Below 64 MB the pairs go through the upload buffer, in as many row blocks
    as they need (1024 rays: a quarter of the entries, the most), and a block
    whose pairs do not fit goes dense (the last rows, with the most rays)."""
    n = 4096 - 8  # 64 MB less a little
    faces = np.concatenate([scenes.icosphere(4, 1.0, inward=True)] * 2)[:n]
    front, zero = np.full(n, rays if rays < 1000 else rays - 3, np.int32), np.zeros(n, np.int32)
    uneven = np.where(np.arange(n) < 3000, 20, 3 * rays).astype(np.int32)
    c = native.Context(0)
    _limit(c, 1)
    c.scene_set(faces)
    c.grid_build(cells_per_face=16)
    for k, f in enumerate((front, uneven)):
        threads = c.host_threads()
        got = c.form_factor_counts(f, zero, 5)
        moved = c.stats().d2h_bytes
        assert moved < 4 * n * n  # packed, or (the last block) in part
        assert k or moved < 4 * rays * n + (1 << 20)
        c.set_host_threads(0)
        assert np.array_equal(got, c.form_factor_counts(f, zero, 5))
        assert c.stats().d2h_bytes == 4 * n * n
        c.set_host_threads(threads)
