"""Host outputs of 16 to 64 MB, which move as pairs in row blocks like the larger
ones: pageable, pinned and odd destinations, mesh rows, sparse and dense
matrices (past a quarter of the entries they are copied dense), growing and
shrinking in one context, against the device output.  Tolerance: none."""
import numpy as np
import pytest

from form_factors_b200 import scenes

pytestmark = pytest.mark.gpu


# 2047^2 words lie below 16 MB, 2048^2 are 16 MB
@pytest.mark.parametrize("n", [2047, 2048, 3001, 3700, 2100])
@pytest.mark.parametrize("rays", [1, 40, 3000])
def test_counts_and_factors(ctx, n, rays):
    import torch
    faces = np.concatenate([scenes.icosphere(4, 1.0, inward=True)[::2], scenes.enclosure(3, 11)])[:n]
    n = len(faces)
    ctx.scene_set(faces)
    ctx.grid_build(cells_per_face=64, skip_empty=True)
    front, rear = np.full(n, rays, np.int32), np.zeros(n, np.int32)
    front[::9], rear[::5] = 0, 2
    want = torch.empty((n, n), dtype=torch.int32, device="cuda")
    ctx.form_factor_counts(front, rear, 11, epoch=rays, out=want)
    ctx.synchronize()
    want = want.cpu().numpy().view(np.uint32)
    got = np.full((n, n), 0xDEADBEEF, np.uint32)
    ctx.form_factor_counts(front, rear, 11, epoch=rays, out=got)
    assert np.array_equal(got, want)
    raw = torch.full((n * n + 1,), -1, dtype=torch.int32, pin_memory=True)
    ctx.form_factor_counts(front, rear, 11, epoch=rays, out=raw[1:])
    assert np.array_equal(raw[1:].numpy().view(np.uint32).reshape(n, n), want)
    ff = ctx.form_factors(front, rear, 11, epoch=rays)
    with np.errstate(divide="ignore", invalid="ignore"):
        ref = want.astype(np.float32) * (np.float32(1) / (front + rear).astype(np.float32))[:, None]
    nan = np.isnan(ref)
    assert np.array_equal(np.isnan(ff), nan) and np.array_equal(ff[~nan].view(np.uint32), ref[~nan].view(np.uint32))
    rows = (np.arange(n) * 7 % n).astype(np.int32)  # faces in another order
    ctx.form_factor_counts(front, rear, 11, epoch=rays, face_to_row=rows, n_rows=n, out=got)
    by_row = np.zeros((n, n), np.uint32)
    np.add.at(by_row, (rows[:, None], rows[None, :]), want)
    assert np.array_equal(got, by_row)
