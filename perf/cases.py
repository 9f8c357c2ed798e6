"""Workloads of the form-factor path as a user's program calls it, for timing and comparing builds.

Each case is one pass through the public entry points of form_factors_b200:
a new scene solved from its faces, a resident scene traced again with a new
seed, rays emitted and cast in the reference's call order, the two ray-traced
thermal equations, the matrix written as CSV text, a batch of scenes, and an
OBJ scene taken from its text to form factors.  Scenes and sizes are those of
the package's scene generators, tests and benchmark.
"""
import functools
import math

import numpy as np
import torch

from form_factors_b200 import emission, native, scenes

FIXED_SCENES = ("box", "enclosure")  # geometry that does not depend on the seed


def listed():
    return [
        # The smallest solve: the closed box of 12 triangles, new faces to
        # host matrix.  Launches, copies and host work are all of its time.
        dict(name="box_solve", kind="solve", scene="box", faces=12, rays=1000, sided=2, cells=0, stats=True),
        # Two parallel unit squares of 200 triangles each with many rays per
        # face through a 16^3 grid: a small matrix whose entries repeat.
        dict(name="plates_counts", kind="counts", scene="plates", faces=400, rays=100000, sided=1, grid=16,
             tuned=False, stats=False, out="device"),
        # The closed enclosure of the benchmark: 22 080 faces, 1000 rays per
        # face, the 1.95 GB matrix resident, grid and launch shape tuned.
        dict(name="enclosure_counts", kind="counts", scene="enclosure", faces=22080, rays=1000, sided=1, grid=0,
             tuned=True, stats=False, out="device"),
        # The same solve delivered to page-locked host memory, end to end.
        dict(name="enclosure_host", kind="counts", scene="enclosure", faces=22080, rays=1000, sided=1, grid=0,
             tuned=True, stats=False, out="host"),
        # Occluded clutter whose geometry changes before every solve (a
        # moving scene): upload, grid build, trace, host form factors.  All
        # options at their defaults.
        dict(name="clutter_solve", kind="solve", scene="clutter", faces=4028, rays=1000, sided=1, cells=0,
             stats=True),
        # Form factors between meshes (the reference's matrix is per mesh):
        # both sides emit, faces of a mesh share a row, floats stay on the
        # device.
        dict(name="enclosure_meshes", kind="meshes", scene="enclosure", faces=22080, rays=430, sided=2, per_mesh=20,
             stats=False),
        # The reference's unfused call order: rays materialised by the
        # emission system, then cast with hit points by the caster.
        dict(name="clutter_cast", kind="cast", scene="clutter", faces=4028, rays=601, sided=1, cells=0, stats=True),
        # One step of the radiance equation over per-face meshes.
        dict(name="enclosure_radiance", kind="radiance", scene="enclosure", faces=22080, rays=1000, per_mesh=1,
             cells=192, stats=True),
        # One step of the distant-source equation (a disc of parallel rays).
        dict(name="sphere_source", kind="source", scene="sphere", faces=20000, rays=10000000, per_mesh=100,
             cells=64, stats=True),
        # CSV text of the enclosure's matrix from its resident counts.
        dict(name="enclosure_csv", kind="csv", scene="enclosure", faces=22080, rays=1000, sided=1, floats=False),
        # Independent scenes of uneven size in one batched launch.
        dict(name="batch_mixed", kind="batch", scenes=24, n_min=200, n_max=10000, rays=1500),
        # An OBJ scene from its text to form factors between its objects.
        dict(name="obj_solve", kind="obj", scene="clutter", faces=100000, rays=20, per_mesh=1000, edge=0.02,
             stats=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "counts", "counts", "counts", "meshes", "cast", "radiance", "source", "csv", "batch",
                       "obj"])
    scene = rng.choice(["plates", "sphere", "clutter"])
    sided = rng.choice([1, 1, 2])
    if kind == "solve":
        n = _log(rng, 24, 6000)
        return dict(kind=kind, scene=scene, faces=n, rays=_log(rng, 50, min(20000, 8000000 // n)), sided=sided,
                    cells=rng.choice([0, 0, 64, 128]), stats=rng.choice([True, False]))
    if kind == "counts":
        n = _log(rng, 100, 20000)
        out = rng.choice(["device", "device", "host"])
        return dict(kind=kind, scene=scene, faces=n, rays=_log(rng, 50, min(100000, 20000000 // n)), sided=sided,
                    grid=rng.choice([0, 0, rng.randint(8, 120)]), tuned=False, stats=rng.choice([True, False]),
                    out=out)
    if kind == "meshes":
        n = _log(rng, 400, 20000)
        return dict(kind=kind, scene=scene, faces=n, rays=_log(rng, 50, 10000000 // n), sided=sided,
                    per_mesh=rng.randint(2, 40), stats=rng.choice([True, False]))
    if kind == "cast":
        n = _log(rng, 200, 6000)
        return dict(kind=kind, scene=scene, faces=n, rays=_log(rng, 10, min(4000, 2500000 // n)), sided=sided,
                    cells=rng.choice([0, 64, 128]), stats=True)
    if kind == "radiance":
        n = _log(rng, 200, 20000)
        return dict(kind=kind, scene=scene, faces=n, rays=_log(rng, 50, 15000000 // n),
                    per_mesh=rng.choice([1, 1, rng.randint(2, 30)]), cells=rng.choice([0, 64, 192]),
                    stats=rng.choice([True, False]))
    if kind == "source":
        n = _log(rng, 200, 20000)
        return dict(kind=kind, scene=scene, faces=n, rays=_log(rng, 100000, 10000000), per_mesh=rng.randint(1, 100),
                    cells=rng.choice([0, 64, 128]), stats=rng.choice([True, False]))
    if kind == "csv":
        n = _log(rng, 100, 8000)
        return dict(kind=kind, scene=scene, faces=n, rays=_log(rng, 50, min(20000, 8000000 // n)), sided=sided,
                    floats=rng.choice([True, False]))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(5, 30), n_min=200, n_max=_log(rng, 1000, 9000),
                    rays=_log(rng, 200, 1500))
    return dict(kind=kind, scene="clutter", faces=_log(rng, 2000, 90000), rays=_log(rng, 10, 40),
                per_mesh=rng.randint(50, 1500), edge=0.02, stats=rng.choice([True, False]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _fixed(scene):
    return scenes.enclosure(5, 20) if scene == "enclosure" else scenes.unit_box()


def _faces(case, seed):
    """The scene's faces: clutter drawn from the seed, spheres turned by a
    random rotation, the others fixed (their rays differ by seed)."""
    if case["scene"] in FIXED_SCENES:
        return _fixed(case["scene"])
    rng = np.random.default_rng(seed)
    if case["scene"] == "clutter" and "edge" in case:
        k = max(1, int(round(math.sqrt(case["faces"] / 48.0))))
        return scenes.clutter(case["faces"] - 12 * k * k, case["edge"], seed=int(rng.integers(1 << 31)),
                              enclosure_cells=k)
    if case["scene"] == "clutter" and case["faces"] == 4028:
        return scenes.clutter(2000, 0.05, seed=int(rng.integers(1 << 31)), enclosure_cells=13)
    f = scenes.family_scene(case["scene"], case["faces"], rng)
    if case["scene"] == "sphere":
        f = scenes.transform(f, rot=scenes.random_rotations(rng, 1)[0])
    return f


def _ray_counts(case, faces):
    """(front, rear) rays per face: a fixed front count, or the reference's
    area-weighted budget over both sides."""
    n = len(faces)
    if case["sided"] == 1:
        return emission.front_only(n, case["rays"])
    w, total = emission.two_sided_weights(faces)
    return emission.ray_counts(2 * case["rays"] * n, w, total)


def _mesh_rows(n, per_mesh):
    return (np.arange(n) // per_mesh).astype(np.int32)


def _mesh_table(n, per_mesh):
    first = np.arange(0, n, per_mesh)
    m = np.zeros((len(first), 3), np.int32)
    m[:, 0] = first
    m[:, 1] = np.minimum(first + per_mesh, n) - first
    m[:, 2] = np.arange(len(first)) % 2
    return m


MATERIALS = np.array([(0.9, 0.0, 0.8, 0.8), (0.7, 0.6, 0.5, 0.4)], np.float32)  # emissivities, absorbances


def _obj_text(faces, per_object):
    """OBJ text of the faces, one object per `per_object` of them, and the
    coordinates as written."""
    out = []
    v = faces.reshape(-1, 3)
    for k in range(0, len(faces), per_object):
        e = min(len(faces), k + per_object)
        m = 3 * (e - k)
        out.append("o part_%d\n" % (k // per_object))
        out.append(("v %.9g %.9g %.9g\n" * m) % tuple(v[3 * k:3 * e].ravel().tolist()))
        out.append(("f %d %d %d\n" * (e - k)) % tuple(range(3 * k + 1, 3 * e + 1)))
    return "".join(out).encode()


def _batch(case):
    sl, _ = scenes.batch_workload(case["scenes"], case["n_min"], case["n_max"], 1000, 2000, seed=case["scenes"])
    rng = np.random.default_rng(case["rays"])
    rays = rng.integers(max(1, case["rays"] // 4), case["rays"] * 2, len(sl))
    return sl, rays


class State:
    pass


def prepare(case, seed):
    s = State()
    s.kind, s.seed = case["kind"], int(seed) * 1000003 + 12345
    s.ctx = native.Context(torch.cuda.current_device())
    ctx = s.ctx
    if not case.get("stats", False):
        ctx.set_stats(False)
    if s.kind == "batch":
        s.scenes, rays = _batch(case)
        s.front = np.concatenate([np.full(len(f), r, np.int32) for f, r in zip(s.scenes, rays)])
        ctx.batch_set(s.scenes, cells_per_face=64.0)
        ctx.batch_prepare(s.front, np.zeros_like(s.front), np.arange(1, len(s.scenes) + 1) * 7919 + s.seed)
        s.offsets, words = ctx.batch_counts_layout()
        s.counts = torch.empty(words, dtype=torch.int32, device="cuda")  # uint32 bit patterns
        return s
    s.faces = _faces(case, seed)
    n = len(s.faces)
    if s.kind == "obj":
        s.text = _obj_text(s.faces, case["per_mesh"])
        s.front, s.rear = emission.front_only(n, case["rays"])
        s.faces = None
        return s
    if s.kind in ("radiance", "source"):
        s.meshes, s.rays = _mesh_table(n, case["per_mesh"]), int(case["rays"])
        if s.kind == "radiance":
            s.rays *= n
            s.temperatures = _temperatures(len(s.meshes), seed)
        ctx.scene_set(s.faces)
        ctx.grid_build(cells_per_face=case["cells"] or None)
        return s
    s.front, s.rear = _ray_counts(case, s.faces)
    if s.kind == "solve":
        s.cells = case["cells"] or None
        s.out = np.empty((n, n), np.float32)
        return s
    ctx.scene_set(s.faces)
    if case.get("tuned"):
        ctx.autotune(s.front, s.rear, seed=1, candidates=[dict(cells_per_face=c) for c in (128.0, 192.0, 256.0)])
    elif case.get("grid"):
        ctx.grid_build(dims=(case["grid"],) * 3)
    else:
        ctx.grid_build(cells_per_face=case.get("cells") or None)
    if s.kind == "meshes":
        s.rows = _mesh_rows(n, case["per_mesh"])
        s.n_rows = int(s.rows[-1]) + 1
        s.outgoing = np.bincount(s.rows, weights=s.front.astype(np.int64) + s.rear).astype(np.int32)
        s.out = torch.empty((s.n_rows, s.n_rows), dtype=torch.float32, device="cuda")
    elif s.kind == "cast":
        total = int(s.front.sum(dtype=np.int64) + s.rear.sum(dtype=np.int64))
        s.rays = torch.empty((total, 6), dtype=torch.float32, device="cuda")
        s.hit = torch.empty(total, dtype=torch.int32, device="cuda")
        s.points = torch.empty((total, 3), dtype=torch.float32, device="cuda")
    elif s.kind == "csv":
        counts = torch.empty((n, n), dtype=torch.int32, device="cuda")
        ctx.form_factor_counts(s.front, s.rear, s.seed, n_rows=n, out=counts)
        outgoing = s.front + s.rear
        if case["floats"]:
            s.matrix = dict(ff=torch.empty((n, n), dtype=torch.float32, device="cuda"))
            ctx.normalise(counts, outgoing, out=s.matrix["ff"])
            ctx.synchronize()
        else:
            s.matrix = dict(counts=counts, outgoing=torch.from_numpy(outgoing).cuda())
        # room for any matrix of this many rays: 2 bytes per zero, at most 13 for another entry
        cap = 2 * n * n + 11 * min(n * n, int(s.front.sum(dtype=np.int64) + s.rear.sum(dtype=np.int64)))
        s.text = torch.zeros(cap, dtype=torch.uint8, device="cuda")
    elif case["out"] == "host":
        s.out = torch.empty((n, n), dtype=torch.int32, pin_memory=True)
    else:
        s.out = torch.empty((n, n), dtype=torch.int32, device="cuda")
    s.n = n
    return s


def _temperatures(n, seed):
    return (300.0 + 100.0 * np.random.default_rng(seed).random(n)).astype(np.float32)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    ctx = s.ctx
    if s.kind == "solve":
        ctx.scene_set(s.faces)
        ctx.grid_build(cells_per_face=s.cells)
        return ctx.form_factors(s.front, s.rear, s.seed, out=s.out)
    if s.kind == "counts":
        return ctx.form_factor_counts(s.front, s.rear, s.seed, n_rows=s.n, out=s.out)
    if s.kind == "meshes":
        return ctx.form_factors(s.front, s.rear, s.seed, face_to_row=s.rows, n_rows=s.n_rows, outgoing=s.outgoing,
                                out=s.out)
    if s.kind == "cast":
        ctx.emit(s.front, s.rear, s.seed, out=s.rays)
        ctx.cast(s.rays, hit=s.hit, points=s.points)
        return dict(rays=s.rays, hit=s.hit, points=s.points)
    if s.kind == "radiance":
        e, a = ctx.radiance_step(s.faces, s.meshes, MATERIALS, s.temperatures, s.rays, s.seed)
        return dict(emission=e, absorption=a)
    if s.kind == "source":
        return ctx.distant_source_step(s.faces, s.meshes, MATERIALS, s.rays, 1361.0, [0.3, -0.4, -0.8], s.seed)
    if s.kind == "csv":
        return dict(length=ctx.csv_format(out=s.text, **s.matrix), text=s.text)
    if s.kind == "batch":
        ctx.batch_launch(s.counts, s.offsets, advance_epoch=False)
        return s.counts
    info = ctx.obj_parse(s.text)
    faces, meshes, _ = ctx.obj_result(info)
    ctx.obj_scene_set(info["n_faces"])
    ctx.grid_build()
    rows = np.repeat(np.arange(len(meshes), dtype=np.int32), meshes[:, 1])
    ff = ctx.form_factors(s.front, s.rear, s.seed, face_to_row=rows, n_rows=len(meshes))
    return dict(faces=faces, meshes=meshes, form_factors=ff)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _size(case):
    """Number of faces of the case's scene."""
    return len(_faces(case, 0))


def work(case):
    """Bytes read and written once, and the arithmetic of the method: per
    traced ray one emission (about 60 operations) and the one test of the
    triangle it hits (42, math/triangle.cpp:40-78)."""
    kind = case["kind"]
    if kind == "batch":
        sl, rays = _batch(case)
        n = sum(len(f) for f in sl)
        return {"bytes": 4.0 * sum(len(f) ** 2 for f in sl) + 44.0 * n,
                "flops": 102.0 * sum(len(f) * int(r) for f, r in zip(sl, rays))}
    n = _size(case)
    if kind == "radiance":
        rays = case["rays"] * n
        return {"bytes": 36.0 * n + 24.0 * (n // case["per_mesh"]), "flops": 102.0 * rays}
    if kind == "source":
        return {"bytes": 36.0 * n + 16.0 * (n // case["per_mesh"]), "flops": 92.0 * case["rays"]}
    rays = case["rays"] * n * case.get("sided", 1)
    if kind == "csv":
        nonzero = min(n * n, rays)
        return {"bytes": 4.0 * n * n + 2.0 * n * n + 5.0 * nonzero, "flops": 40.0 * nonzero}
    if kind == "cast":
        return {"bytes": (24.0 + 24.0 + 16.0) * rays + 36.0 * n, "flops": 102.0 * rays}
    if kind == "obj":
        return {"bytes": 120.0 * n + 36.0 * n + 4.0 * (n / case["per_mesh"]) ** 2, "flops": 102.0 * rays}
    rows = n / case["per_mesh"] if kind == "meshes" else n
    return {"bytes": 4.0 * rows * rows + 44.0 * n, "flops": 102.0 * rays}


# ---------------------------------------------------------------------------
# the same values in 64 bits
# ---------------------------------------------------------------------------
def _philox(c, k0, k1):
    """Philox4x32-10 on four uint64 arrays of 32-bit words."""
    low = np.uint64(0xFFFFFFFF)
    x, y, z, w = c
    for _ in range(10):
        p0, p1 = x * np.uint64(0xD2511F53), z * np.uint64(0xCD9E8D57)
        x, y, z, w = ((p1 >> np.uint64(32)) ^ y ^ np.uint64(k0), p1 & low,
                      (p0 >> np.uint64(32)) ^ w ^ np.uint64(k1), p0 & low)
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return x, y, z, w


def _emit64(faces, front, rear, seed):
    """Malley rays (origin, end point) of every face in float64."""
    per = front.astype(np.int64) + rear
    f = np.repeat(np.arange(len(faces)), per)
    j = np.arange(len(f)) - np.repeat(np.cumsum(per) - per, per)
    zero = np.zeros(len(f), np.uint64)
    draws = _philox((j.astype(np.uint64), f.astype(np.uint64), zero, zero + np.uint64(0x46464231)),
                    seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF)
    a, b, r, phi = [(d >> np.uint64(8)).astype(np.float64) / 2.0 ** 24 for d in draws]
    over = (a.astype(np.float32) + b.astype(np.float32)) > 1
    a, b = np.where(over, 1 - a, a), np.where(over, 1 - b, b)
    p = faces.reshape(-1, 3, 3).astype(np.float64)
    e1, e2 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    nrm = np.cross(e1, e2)
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    origin = p[f, 0] + e1[f] * a[:, None] + e2[f] * b[:, None]
    x, y = np.sqrt(r) * np.cos(2 * np.pi * phi), np.sqrt(r) * np.sin(2 * np.pi * phi)
    z = np.sqrt(1 - r) * np.where(j >= front[f], -1.0, 1.0)
    # rotation of +z towards the normal: R = I + K + K^2 / (1 + cos), transposed
    # as the reference's row-major product applies it
    c = nrm[:, 2]
    flat = np.hypot(nrm[:, 0], nrm[:, 1]) < 1e-18
    vx, vy = -nrm[:, 1], nrm[:, 0]
    k = np.where(flat, 0.0, 1.0 / np.where(1 + c == 0, 1.0, 1 + c))
    m = np.zeros((len(faces), 3, 3))
    m[:, 0, 0], m[:, 0, 1], m[:, 0, 2] = 1 - k * vy * vy, k * vx * vy, vy
    m[:, 1, 0], m[:, 1, 1], m[:, 1, 2] = k * vx * vy, 1 - k * vx * vx, -vx
    m[:, 2, 0], m[:, 2, 1], m[:, 2, 2] = -vy, vx, np.where(flat, 1.0, 1 - k * (vx * vx + vy * vy))
    back = flat & (c < 0)
    m[back] = np.diag([1.0, -1.0, -1.0])
    d = np.einsum("nij,nj->ni", m[f], np.stack([x, y, z], 1))
    return np.concatenate([origin + 1e-4 * d, origin + d], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "cast":
        faces = _faces(case, seed)
        front, rear = _ray_counts(case, faces)
        # no value for the points: a ray within rounding of an edge hits one
        # triangle or its neighbour, or passes between them, by its last bit
        return dict(rays=torch.from_numpy(_emit64(faces, front, rear, int(seed) * 1000003 + 12345)), hit=None,
                    points=None)
    if kind == "radiance":
        # sigma T^4 (front + rear emissivity) area per mesh; the absorbed
        # power is a Monte Carlo sum over the rays' own hits
        faces = _faces(case, seed).reshape(-1, 3, 3).astype(np.float64)
        meshes = _mesh_table(len(faces), case["per_mesh"])
        area = np.linalg.norm(np.cross(faces[:, 1] - faces[:, 0], faces[:, 2] - faces[:, 0]), axis=1) / 2
        per = np.add.reduceat(area, meshes[:, 0])
        t = _temperatures(len(meshes), seed).astype(np.float64)
        eps = MATERIALS.astype(np.float64)[meshes[:, 2], :2].sum(1)
        return dict(emission=torch.from_numpy(5.6704e-8 * t ** 4 * eps * per), absorption=None)
    if kind == "obj":
        return dict(faces=torch.from_numpy(_faces(case, seed).astype(np.float64)), meshes=None, form_factors=None)
    return None  # counts and text are whole numbers; a form factor is a count over a count
