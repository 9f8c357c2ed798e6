"""The one-pass CSV kernel (device buffers) at the edges of its tiles: matrix
sides around the 512 entries of a warp and the 4096 of a block, rows that end
inside a warp or many times in one, empty, sparse and full matrices (a warp's
text in one window or several), every class of float, counts whose rows have no
or a negative number of rays, and text that starts at any byte offset.  The
expected bytes are "%g" of each entry joined by ';' with '\\n' after each row
(csv_export::export_csv, import_export/csv_export.cpp:26-46).  Tolerance: none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _text(ff):
    """The matrix as text; NaNs keep their sign."""
    def g(x, neg):
        return ("-nan" if neg else "nan") if x != x else "%g" % x
    neg = np.signbit(ff)
    return "".join(";".join(g(x, s) for x, s in zip(r, b)) + "\n"
                   for r, b in zip(ff.astype(np.float64).tolist(), neg.tolist())).encode()


def _check(ctx, want, offset, **source):
    import torch
    buf = torch.full((len(want) + offset + 64,), 35, dtype=torch.uint8, device="cuda")
    n = ctx.csv_format(out=buf[offset:offset + len(want)], **source)
    got = buf.cpu().numpy()
    assert n == len(want)
    text = got[offset:offset + n].tobytes()
    if text != want:
        at = next(i for i, (a, b) in enumerate(zip(text, want)) if a != b)
        raise AssertionError("byte %d: got %r want %r" % (at, text[max(0, at - 20):at + 20], want[max(0, at - 20):at + 20]))
    assert (got[:offset] == 35).all() and (got[offset + n:] == 35).all()
    assert ctx.csv_length(**source) == n


@pytest.mark.parametrize("n", [1, 2, 7, 31, 64, 181, 511, 512, 513, 700, 1025])
@pytest.mark.parametrize("density", [0.0, 0.04, 0.4, 1.0])
def test_floats(ctx, n, density):
    import torch
    rng = np.random.default_rng(n + int(100 * density))
    ff = np.zeros((n, n), np.float32)
    m = rng.random((n, n)) < density
    k = int(m.sum())
    kinds = rng.integers(0, 8, k)
    v = rng.integers(0, 2 ** 32, k, dtype=np.uint64).astype(np.uint32).view(np.float32)  # any float
    form = (rng.integers(1, 40, k) * (np.float32(1) / rng.integers(1, 5000, k).astype(np.float32))).astype(np.float32)
    edge = rng.choice(np.array([-0.0, np.inf, -np.inf, 1e-4, 9.99999e-5, 999999.5, 1e6, 0.5, 1, 100000, 1e-45], np.float32), k)
    v = np.where(kinds < 5, form, np.where(kinds < 7, v, edge)).astype(np.float32)
    ff[m] = v
    _check(ctx, _text(ff), n % 16, ff=torch.from_numpy(ff).cuda())


@pytest.mark.parametrize("n", [1, 5, 33, 512, 600, 1100])
@pytest.mark.parametrize("rays", [3, 1000])
def test_counts(ctx, n, rays):
    import torch
    rng = np.random.default_rng(n * rays)
    counts = rng.poisson(min(1.0, rays / n) * 0.5, (n, n)).astype(np.uint32)
    outgoing = np.maximum(counts.sum(1), 1).astype(np.int32)
    outgoing[::7] = rays
    if n > 20:
        outgoing[3], outgoing[11] = 0, -5
    with np.errstate(divide="ignore", invalid="ignore"):
        ff = counts.astype(np.float32) * (np.float32(1) / outgoing.astype(np.float32))[:, None]
    ff = np.where(np.isnan(ff), np.float32(np.nan), ff).astype(np.float32)  # 0 * inf on the GPU is a positive NaN
    _check(ctx, _text(ff), (3 * n) % 16, counts=torch.from_numpy(counts.view(np.int32)).cuda(),
           outgoing=torch.from_numpy(outgoing).cuda())


@pytest.mark.parametrize("n", [1739, 1742, 1793])  # 5 x 148 blocks of 4096 entries: 1741 rows and a part
def test_sizes_around_one_wave(ctx, n):
    """The switch from 128 to 512 entries per warp, sparse rows and full ones."""
    import torch
    rng = np.random.default_rng(n)
    ff = np.zeros((n, n), np.float32)
    m = rng.random((n, n)) < 0.03
    m[5:40] = True
    ff[m] = rng.integers(1, 40, int(m.sum())).astype(np.float32) * np.float32(1 / 997)
    _check(ctx, _text(ff), n % 16, ff=torch.from_numpy(ff).cuda())
