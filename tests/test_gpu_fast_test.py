"""The grid traversal's fast triangle test decides only what its error bounds
leave certain and hands the rest to the reference's float test, so a cast
through any grid equals the brute-force definition (ray_caster/naive_cpu.cpp
:65-97) bit for bit.  Checked here where the bounds, the landing bias or the
box entry could go wrong: scaled and far-off scenes, slivers, flat scenes,
doubled faces (exact ties), one-cell and strongly uneven grids, rays aimed at
vertices and along edges, axis-parallel rays, rays whose end point is very
near or very far, and origins on faces, on the box and far outside it.
Tolerance: none."""
import numpy as np
import pytest

from form_factors_b200 import scenes
import rays as R

pytestmark = pytest.mark.gpu


def _slivers(n, seed):
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.1, 0.9, (n, 3))
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([a, a + 0.6 * d, a + 0.3 * d + rng.normal(scale=2e-3, size=(n, 3))], axis=1).astype(np.float32)


def _scene(name):
    if name == "slivers":
        return np.concatenate([_slivers(150, 5), scenes.unit_box()])
    if name == "flat":
        return scenes.plate_grid(1, 1, 9, 7)
    if name == "doubled":
        f = scenes.clutter(120, 0.15, seed=9, enclosure_cells=3)
        return np.concatenate([f, f[::-1], scenes.flip(f[:40])])
    return scenes.clutter(250, 0.1, seed=3, enclosure_cells=4)


def _rays(faces, rng, n):
    p = faces.reshape(-1, 3, 3).astype(np.float64)
    lo, hi = p.reshape(-1, 3).min(0), p.reshape(-1, 3).max(0)
    size = float(np.linalg.norm(hi - lo))
    f = rng.integers(0, len(faces), n)
    b = rng.dirichlet((1, 1, 1), n)
    on_face = np.einsum("nk,nkj->nj", b, p[f])
    vertex = p[rng.integers(0, len(faces), n), rng.integers(0, 3, n)]
    edge = 0.5 * (p[f, 0] + p[f, 1])
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    box = lo + rng.random((n, 3)) * (hi - lo)
    wall = box.copy()
    axis = rng.integers(0, 3, n)
    wall[np.arange(n), axis] = np.where(rng.random(n) < 0.5, lo[axis], hi[axis])
    unit = np.eye(3)[rng.integers(0, 3, n)] * rng.choice([-1.0, 1.0], n)[:, None]
    k = 0.3 * size
    parts = [(on_face + 1e-4 * d, on_face + d),                # as emitted
             (box, vertex), (box, edge), (vertex, edge),        # at vertices, edges, along edges
             (box, box + k * unit), (on_face, on_face + k * unit), (wall, wall + k * unit), (wall, wall + k * d),
             (box, box + 1e-3 * d), (box, box + 0.05 * d), (box, box + 300.0 * size * d),
             (box - 2.0 * size * d, box), (box - 15.0 * size * d, box - 15.0 * size * d + 0.1 * d),
             (edge, edge + k * (p[f, 1] - p[f, 0]))]
    return np.concatenate([np.concatenate([o, e], 1) for o, e in parts]).astype(np.float32)


@pytest.mark.parametrize("name", ["clutter", "slivers", "flat", "doubled"])
@pytest.mark.parametrize("scale,shift", [(1.0, (0, 0, 0)), (0.3, (0, 0, 0)), (40.0, (0, 0, 0)), (1.0, (90.0, -35.0, 14.0))])
def test_cast_equals_brute_force(ctx, oracle, name, scale, shift):
    faces = scenes.transform(_scene(name) * np.float32(scale), shift=shift)
    rng = np.random.default_rng(17)
    rays = np.concatenate([_rays(faces, rng, 300), R.mixed_rays(rng, faces, 1500)])
    want_hit, want_pts = oracle.cast_naive(faces, rays)
    ctx.scene_set(faces)
    m = want_hit >= 0
    assert m.any()
    for kw in (dict(), dict(dims=(1, 1, 1)), dict(dims=(256, 3, 2)), dict(dims=(2, 31, 256), skip_empty=False),
               dict(cells_per_face=256)):
        ctx.grid_build(**kw)
        hit, pts = ctx.cast(rays)
        bad = np.nonzero(hit != want_hit)[0]
        assert bad.size == 0, "%s: %d of %d hits differ, first %s: got %s want %s" % (
            kw, bad.size, len(rays), bad[:5], hit[bad[:5]], want_hit[bad[:5]])
        assert np.array_equal(pts[m].view(np.uint32), want_pts[m].view(np.uint32)), "%s: hit points differ" % kw
        assert np.isnan(pts[~m]).all()


@pytest.mark.parametrize("name", ["clutter", "slivers", "doubled"])
@pytest.mark.parametrize("scale,flags", [(1.0, 0), (0.3, 0), (40.0, 0), (1.0, 1)])
def test_counts_equal_oracle(ctx, oracle, name, scale, flags):
    faces = _scene(name) * np.float32(scale)
    n = len(faces)
    rng = np.random.default_rng(23)
    front, rear = rng.integers(0, 90, n).astype(np.int32), rng.integers(0, 40, n).astype(np.int32)
    want = oracle.form_factor_counts(faces, front, rear, seed=5, epoch=3, flags=flags)
    ctx.scene_set(faces)
    for kw in (dict(), dict(dims=(3, 200, 5))):
        ctx.grid_build(**kw)
        for stats in (True, False):
            ctx.set_stats(stats)
            got = ctx.form_factor_counts(front, rear, seed=5, epoch=3, flags=flags)
            assert np.array_equal(got, want), "%s stats=%s: %d entries differ" % (kw, stats, (got != want).sum())
        ctx.set_stats(True)
