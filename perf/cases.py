"""The work that users of this framework have it do, as measured cases.

A case is one pass through the public entry points: an extraction through the
pyramid and traversal handles, a batch, a differentiable step, a welded mesh.
Sizes come from the repository's workloads (hpmc_b200/datasets.py), its demos
(hpmc_b200/apps/) and its tests, plus ragged sizes of the same ranges.

  listed()             the cases
  draw(rng)            another case of the same ranges
  prepare(case, seed)  fields, handles and output buffers on the GPU
  run(state)           one pass and its outputs
  work(case)           bytes and operations a pass cannot do without
  exact(case, seed)    the outputs in 64 bits, in plain torch

The scene of a case (where its balls are, how large its volumes are) is the
case's own; a seed moves it a little, as the next frame or the next step of an
optimisation does, and draws the noise.  Vertex buffers are sized once with
some room, as a program sizes them for many frames.

Sizes are (x, y, z) lattice samples; field tensors are (z, y, x).
"""
from __future__ import annotations

import functools
import glob
import math
import random

import numpy as np
import torch

import hpmc_b200 as H
from hpmc_b200 import autograd

DEV = "cuda"
MAX_SAMPLES = 48_000_000  # of a drawn volume


def listed():
    return [
        # The plain small volume, as an interactive program uses it: build, read the count, extract.
        dict(name="metaballs_64", path="handle", field="metaballs", dtype="f32", x=64, y=64, z=64, balls=8, scene=0,
             normals="central", read_count=True),
        # The demos' frame: a functor field in gradient mode, captured as interleaved normals and positions.
        dict(name="functor_feedback_128", path="functor", x=128, y=128, z=128, iso=0.2, read_count=True),
        # A scanned byte volume of odd size read as normalised texture values, the reference's forward normals.
        dict(name="unorm8_odd_253", path="handle", field="noise", dtype="unorm8", x=253, y=231, z=197,
             normals="forward", read_count=True),
        # A byte volume full of ties whose surface fills it: the most vertices per sample.
        dict(name="noise_u8_256", path="handle", field="noise", dtype="u8", x=256, y=256, z=256, normals="central",
             read_count=False),
        # A float volume whose rows are no multiple of 16 bytes.
        dict(name="ragged_f32_301", path="handle", field="cayley", dtype="f32", x=301, y=257, z=129,
             normals="forward", read_count=False),
        # A wide slab, few slices, forward normals.
        dict(name="slab_512x512x33", path="handle", field="cayley", dtype="f32", x=512, y=512, z=33,
             normals="forward", read_count=False),
        # The large single volume.
        dict(name="cayley_512", path="handle", field="cayley", dtype="f32", x=512, y=512, z=512, normals="central",
             read_count=False),
        # An RGBA texture: gradient and value per sample, gradient mode.
        dict(name="rgba_gradient_128", path="handle", field="rgba", dtype="f32x4", x=128, y=128, z=128, balls=8, scene=1,
             normals="central", read_count=True),
        # Many uneven volumes in one call, tuned once.
        dict(name="batch_64", path="batch", dtype="f32", count=64, lo=32, hi=192, multiple=4, scene=3, tune=True,
             read_count=False),
        # Uneven byte volumes of any size, the offsets read after every call.
        dict(name="batch_ragged_u8_24", path="batch", dtype="u8", count=24, lo=20, hi=120, multiple=1, scene=5,
             tune=False, read_count=True),
        # A training step: extraction and the gradient of the vertices with respect to the field.
        dict(name="autograd_spheres_128", path="autograd", field="spheres", dtype="f32", x=128, y=128, z=128, balls=16, scene=4,
             normals="central"),
        # A welded mesh for a renderer or a simulation.
        dict(name="indexed_192", path="indexed", field="metaballs", dtype="f32", x=192, y=192, z=192, balls=16, scene=6,
             normals="central"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _edges(rng, lo, hi, most):
    """Three edges spread over the logarithm of lo..hi, odd ones among them, of at most `most` samples."""
    while True:
        e = [_log_int(rng, lo, hi) for _ in range(3)]
        if rng.random() < 0.4:
            e[0] = max(lo, e[0] // 4 * 4)
        if e[0] * e[1] * e[2] <= most:
            return dict(x=e[0], y=e[1], z=e[2])


def draw(rng):
    normals = rng.choice(["forward", "central"])
    read = rng.random() < 0.5
    scene = dict(balls=rng.randint(4, 24), scene=rng.randint(0, 1 << 30))
    kind = rng.choice(["f32", "f32", "f32", "byte", "byte", "rgba", "functor", "batch", "batch", "autograd", "indexed"])
    if kind == "f32":
        field = rng.choice(["cayley", "metaballs"])
        c = dict(path="handle", field=field, dtype="f32", normals=normals, read_count=read, **_edges(rng, 24, 512, MAX_SAMPLES))
        return dict(c, **scene) if field == "metaballs" else c
    if kind == "byte":
        return dict(path="handle", field="noise", dtype=rng.choice(["u8", "unorm8"]), normals=normals, read_count=read,
                    **_edges(rng, 32, 300, 12_000_000))
    if kind == "rgba":
        return dict(path="handle", field="rgba", dtype="f32x4", normals=normals, read_count=read, **scene,
                    **_edges(rng, 24, 200, 4_000_000))
    if kind == "functor":
        return dict(path="functor", read_count=read, iso=round(rng.uniform(-0.4, 0.7), 3), **_edges(rng, 24, 256, 8_000_000))
    if kind == "batch":
        return dict(path="batch", dtype=rng.choice(["f32", "u8"]), count=rng.randint(4, 64), lo=rng.randint(16, 40),
                    hi=rng.randint(60, 180), multiple=rng.choice([1, 4]), scene=scene["scene"], tune=False,
                    read_count=read)
    if kind == "autograd":
        return dict(path="autograd", field="spheres", dtype="f32", normals=normals, **scene,
                    **_edges(rng, 24, 192, 5_000_000))
    return dict(path="indexed", field="metaballs", dtype="f32", normals=normals, **scene,
                **_edges(rng, 24, 224, 8_000_000))


# ---------------------------------------------------------------------------
# Inputs

def _axis(n, lo, hi):
    return torch.linspace(lo, hi, n, dtype=torch.float64, device=DEV)


def _balls(scene, count, seed, spheres=False):
    """Centres and radii of the scene, each centre moved by the seed."""
    rng = np.random.default_rng(scene)
    c = rng.uniform(0.2, 0.8, size=(count, 3)) + np.random.default_rng([seed, scene]).uniform(-0.01, 0.01, (count, 3))
    r = rng.uniform(0.05, 0.12 if spheres else 0.15, size=count)
    return [(*map(float, ci), float(ri)) for ci, ri in zip(c, r)]


def _metaballs(size, balls):
    x, y, z = (_axis(n, 0, 1) for n in size)
    out = torch.zeros((size[2], size[1], size[0]), dtype=torch.float64, device=DEV)
    for cx, cy, cz, r in balls:
        out += r * r / ((z - cz).square()[:, None, None] + (y - cy).square()[None, :, None] + (x - cx).square())
    return out.float()


def _spheres(size, balls):
    x, y, z = (_axis(n, 0, 1) for n in size)
    out = torch.full((size[2], size[1], size[0]), math.inf, dtype=torch.float64, device=DEV)
    for cx, cy, cz, r in balls:
        d = (z - cz).square()[:, None, None] + (y - cy).square()[None, :, None] + (x - cx).square()
        out = torch.minimum(out, d.sqrt() - r)
    return out.float()


def _cayley(size, gen):
    """16xyz + 4(x^2 + y^2 + z^2) - 1 and noise, slice by slice (a whole float64 volume is not needed)."""
    x, y, z = (_axis(n, -1, 1) for n in size)
    out = torch.empty((size[2], size[1], size[0]), dtype=torch.float32, device=DEV)
    base = 4 * (x.square()[None, :] + y.square()[:, None]) - 1
    xy = 16 * y[:, None] * x[None, :]
    for k in range(0, size[2], 16):
        zz = z[k:k + 16, None, None]
        part = base + xy * zz + 4 * zz * zz
        noise = torch.randn(part.shape, generator=gen, device=DEV, dtype=torch.float32)
        out[k:k + 16] = (part + 1e-3 * noise.double()).float()
    return out


def _noise(size, gen):
    """Smoothed uniform noise (sigma 3 samples, periodic), rescaled to bytes."""
    u = torch.rand((size[2], size[1], size[0]), generator=gen, device=DEV, dtype=torch.float32)
    g = [torch.exp(-2 * (math.pi * 3.0 * torch.fft.fftfreq(n, device=DEV)).square()) for n in size]
    s = torch.fft.rfftn(u) * (g[2][:, None, None] * g[1][None, :, None] * g[0][: size[0] // 2 + 1])
    s = torch.fft.irfftn(s, s=u.shape)
    lo, hi = s.min(), s.max()
    return torch.round((s - lo) * (255.0 / (hi - lo))).to(torch.uint8)


def _rgba(size, balls):
    """Value and gradient of a sum of soft balls: channels gradient x, y, z, value."""
    x, y, z = (_axis(n, 0, 1) for n in size)
    out = torch.zeros((size[2], size[1], size[0], 4), dtype=torch.float64, device=DEV)
    for cx, cy, cz, r in balls:
        dx, dy, dz = (x - cx)[None, None, :], (y - cy)[None, :, None], (z - cz)[:, None, None]
        d2 = dx * dx + dy * dy + dz * dz + 1e-4
        for i, d in enumerate((dx, dy, dz)):
            out[..., i] -= 2 * r * r * d / d2.square()
        out[..., 3] += r * r / d2
    return out.float()


def _size(case):
    return case["x"], case["y"], case["z"]


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _volume(case, seed):
    """(field, iso) of one volume."""
    size, kind = _size(case), case["field"]
    if kind == "cayley":
        return _cayley(size, _generator(seed)), 0.0
    if kind == "noise":
        return _noise(size, _generator(seed)), 128.0 / 255.0 if case["dtype"] == "unorm8" else 128.0
    balls = _balls(case["scene"], case["balls"], seed, kind == "spheres")
    if kind == "spheres":
        return _spheres(size, balls), 0.0
    return (_rgba if kind == "rgba" else _metaballs)(size, balls), 1.0


def _batch_sizes(case):
    rng = random.Random(case["scene"])
    m = case["multiple"]
    return [max(16, min(case["hi"], m * round(_log_int(rng, case["lo"], case["hi"]) / m))) for _ in range(case["count"])]


def _batch_volumes(case, seed):
    rng = np.random.default_rng(case["scene"])
    fields, isos = [], []
    for n in _batch_sizes(case):
        f = _metaballs((n, n, n), _balls(int(rng.integers(1 << 30)), int(rng.integers(4, 33)), seed))
        iso = float(rng.uniform(0.8, 1.5))
        if case["dtype"] == "u8":
            f, iso = torch.clamp(torch.round(f * 60.0), 0, 255).to(torch.uint8), float(round(iso * 60.0))
        fields.append(f)
        isos.append(iso)
    return fields, isos


def _functor_iso(case, seed):
    """The demos' iso-value changes from frame to frame."""
    return float(np.float32(case["iso"] + np.random.default_rng(seed).uniform(-0.005, 0.005)))


def _cotangents(n, seed):
    g = _generator(seed + 1_000_003)
    return tuple(torch.randn((n, 4), generator=g, device=DEV) for _ in range(2))


# ---------------------------------------------------------------------------
# Preparation and the passes

MODES = {"forward": H.NORMALS_FORWARD, "central": H.NORMALS_CENTRAL}


_CAPACITY = {}


def _key(case):
    return repr(sorted((k, v) for k, v in case.items() if k != "name"))


def _capacity(case, what, count):
    """Rows of a vertex or index buffer: those of seed 0 (count(0)) and some
    room, once per case; a program that meets more vertices makes it anew."""
    k = (_key(case), what)
    if k not in _CAPACITY:
        _CAPACITY[k] = int(1.2 * count(0)) + 4096
    return _CAPACITY[k]


def _zeros(rows, columns=4):
    return torch.zeros((rows, columns), dtype=torch.float32, device=DEV)


def _pyramid(case, field):
    hp = H.HistoPyramid(H.default_constants())
    hp.set_stream(torch.cuda.current_stream())
    if case["path"] == "functor":
        hp.set_lattice_size(*_size(case))
        hp.set_field_custom("hpmc:cayley", gradient=True)
    elif case["dtype"] == "f32x4":
        hp.set_lattice_size(*_size(case))
        name = H.register_device_field(field)
        hp.set_field_texture3d(name, gradient=True)
        H.unregister_device_field(name)  # the pyramid has taken the field over
    else:
        hp.set_field_device(field, unorm=case["dtype"] == "unorm8")
    hp.set_normal_mode(MODES[case.get("normals", "forward")])
    return hp


def _built(case, seed):
    """(field, iso, pyramid) after a first build."""
    field, iso = (None, _functor_iso(case, seed)) if case["path"] == "functor" else _volume(case, seed)
    hp = _pyramid(case, field)
    hp.build(iso)
    return field, iso, hp


def _batch_of(case, seed):
    b = H.Batch(*_batch_volumes(case, seed), normals=H.NORMALS_CENTRAL)
    none = _zeros(1)
    b.extract(none, none, 0)
    return b, b.offsets(allow_truncation=True)[-1]


def _vertices(case, seed):
    if case["path"] == "batch":
        return _batch_of(case, seed)[1]
    return _built(case, seed)[2].acquire_number_of_vertices()


def _welded(case, seed):
    hp = _built(case, seed)[2]
    n = hp.acquire_number_of_vertices()
    pos, nrm = _zeros(n + 1), _zeros(n + 1)
    return H.TraversalHandle(hp).extract_indexed(pos, nrm, torch.zeros(n + 1, dtype=torch.int32, device=DEV))[0]


def prepare(case, seed):
    path = case["path"]
    s = dict(path=path, read_count=case.get("read_count", False))
    if path == "autograd":
        field, iso, hp = _built(case, seed)
        w, u = _cotangents(hp.acquire_number_of_vertices(), seed)
        return dict(s, field=field.requires_grad_(True), iso=iso, normals=MODES[case["normals"]], w=w, u=u)
    rows = _capacity(case, "vertices", functools.partial(_vertices, case))
    if path == "batch":
        b, n = _batch_of(case, seed)
        s.update(batch=b, pos=_zeros(rows), nrm=_zeros(rows))
        if case["tune"]:
            b.autotune(s["pos"], s["nrm"])
    else:
        field, iso, hp = _built(case, seed)
        n = hp.acquire_number_of_vertices()
        th = H.TraversalHandle(hp)
        s.update(hp=hp, th=th, iso=iso, field=field)
        if path == "functor":
            s["feedback"] = _zeros(rows, 6)
            th.set_feedback_buffer(s["feedback"])
        elif path == "indexed":
            s["indices"] = torch.zeros(rows, dtype=torch.int32, device=DEV)
            unique = _capacity(case, "welded", functools.partial(_welded, case))
            s.update(pos=_zeros(unique), nrm=_zeros(unique))
        else:
            s.update(pos=_zeros(rows), nrm=_zeros(rows))
            th.set_buffers(s["pos"], s["nrm"])
    if n > rows:
        raise RuntimeError("the vertex buffers are too small for this seed")
    return s


def run(s):
    path = s["path"]
    if path == "batch":
        s["batch"].extract(s["pos"], s["nrm"])
        offsets = s["batch"].offsets() if s["read_count"] else None
        return {"pos": s["pos"], "nrm": s["nrm"], "offsets": offsets}
    if path == "autograd":
        pos, nrm = autograd.extract(s["field"], s["iso"], normals=s["normals"])
        (grad,) = torch.autograd.grad([pos, nrm], s["field"], [s["w"], s["u"]])
        return {"grad": grad, "count": pos.shape[0]}
    hp, th = s["hp"], s["th"]
    hp.build(s["iso"])
    if path == "indexed":
        counts = th.extract_indexed(s["pos"], s["nrm"], s["indices"])
        return {"pos": s["pos"], "nrm": s["nrm"], "indices": s["indices"], "counts": counts}
    n = hp.acquire_number_of_vertices() if s["read_count"] else None
    if path == "functor":
        th.extract_feedback()
        return {"feedback": s["feedback"], "count": n}
    th.extract()
    return {"pos": s["pos"], "nrm": s["nrm"], "count": n}


# ---------------------------------------------------------------------------
# The same in 64 bits, in plain torch

@functools.lru_cache(maxsize=None)
def _case_tables():
    """Marching-cubes tables as the golden fixtures list them: vertices per
    case, edge of a case's k-th vertex, lower end and axis of each edge."""
    count, edges, ends = np.zeros(256, np.int64), np.zeros((256, 16), np.int64), {}
    files = sorted(glob.glob("tests/golden/*.npz"))
    if not files:
        return None
    for path in files:
        d = np.load(path)
        edges[d["code"], d["k"]] = d["edge"]
        np.maximum.at(count, d["code"], d["k"].astype(np.int64) + 1)
        if not path.endswith("normal_grid.npz"):
            continue
        at = d["pos_fwd"] * np.array(d["codes"].shape[::-1]) - d["cell"]
        inner = (d["t_fwd"] > 0.05) & (d["t_fwd"] < 0.95)
        for e, p in zip(d["edge"][inner], at[inner]):
            axis = int(np.argmax(np.abs(p - np.round(p))))
            p = np.round(p).astype(int)
            p[axis] = 0
            ends[int(e)] = (*map(int, p), axis)
    to = functools.partial(torch.tensor, device=DEV)
    return to(count), to(edges), to([ends[e] for e in range(12)])


def _spread(v):
    for s, m in ((16, 0x0000FFFF0000FFFF), (8, 0x00FF00FF00FF00FF), (4, 0x0F0F0F0F0F0F0F0F), (2, 0x3333333333333333),
                 (1, 0x5555555555555555)):
        v = (v | (v << s)) & m
    return v


def _soup(below):
    """(a, axis) of every vertex in output order, from the samples below the iso-value."""
    count, edges, ends = _case_tables()
    cz, cy, cx = (n - 1 for n in below.shape)
    code = torch.zeros((cz, cy, cx), dtype=torch.uint8, device=DEV)
    for i in range(8):
        dx, dy, dz = i & 1, i >> 1 & 1, i >> 2
        code |= below[dz:dz + cz, dy:dy + cy, dx:dx + cx].to(torch.uint8) << i
    z, y, x = torch.nonzero((code != 0) & (code != 255), as_tuple=True)
    c = code[z, y, x].long()
    del code
    # the tiled 2-D base level: slice z is tile (z mod lx, z div lx), vertices in the Morton order of the tiling
    tx, ty = (1 << max(0, math.ceil(math.log2(n / 2))) for n in (cx, cy))
    lx = 1 << max(0, math.ceil(math.log2(math.sqrt(cz / (tx / ty)))))
    ly = -(-cz // lx)
    size = 1 << math.ceil(math.log2(max(tx * lx, ty * ly)))
    lx = size // tx
    order = torch.argsort(_spread(2 * tx * (z % lx) + x) | _spread(2 * ty * (z // lx) + y) << 1)
    x, y, z, c = x[order], y[order], z[order], c[order]
    n = count[c]
    k = torch.arange(int(n.sum()), device=DEV) - torch.repeat_interleave(torch.cumsum(n, 0) - n, n)
    end = ends[edges[torch.repeat_interleave(c, n), k]]
    return torch.repeat_interleave(torch.stack((x, y, z), 1), n, dim=0) + end[:, :3], end[:, 3]


def _geometry(field, iso, a, axis, central):
    """Positions and normals on a field of 64-bit samples, clamped at its edges."""
    fz, fy, fx = field.shape
    cells = torch.tensor([fx - 1, fy - 1, fz - 1], dtype=torch.float64, device=DEV)
    unit = torch.eye(3, dtype=torch.int64, device=DEV)
    b = a + unit[axis]
    flat = field.reshape(-1)

    def at(p):
        return flat[(p[:, 2].clamp(0, fz - 1) * fy + p[:, 1].clamp(0, fy - 1)) * fx + p[:, 0].clamp(0, fx - 1)]

    t = (at(a) - iso) / (at(a) - at(b))
    n = []
    for e in unit:
        ga, gb = (at(a + e) - at(a - e), at(b + e) - at(b - e)) if central else (at(a + e), at(b + e))
        g = ga + t * (gb - ga)
        n.append(-0.5 * g if central else iso - g)
    p = (a.double() + t[:, None] * unit[axis].double()) / cells
    return p, torch.stack(n, 1) / cells


def _rows(v, rows):
    """`v` in a buffer of `rows` rows, the others zero."""
    out = torch.zeros((rows, *v.shape[1:]), dtype=v.dtype, device=DEV)
    out[: v.shape[0]] = v
    return out


def _streams(p, n, rows):
    """The two vertex streams: positions with w = 1, normals with w = 0."""
    return {k: _rows(torch.cat((v, torch.full((v.shape[0], 1), w, dtype=v.dtype, device=DEV)), 1), rows)
            for k, v, w in (("pos", p, 1.0), ("nrm", n, 0.0))}


def _samples(case, field):
    """The 32-bit values the field stands for."""
    return field.float() / 255.0 if case.get("dtype") == "unorm8" else field.float()


def _gradient_mode(value, grad, iso, central):
    """Positions and normals in gradient mode: the gradients given at the samples."""
    a, axis = _soup(value < iso)
    fz, fy, fx = value.shape
    unit = torch.eye(3, dtype=torch.int64, device=DEV)
    b = a + unit[axis]
    cells = torch.tensor([fx - 1, fy - 1, fz - 1], dtype=torch.float64, device=DEV)
    va, vb = (value[p[:, 2], p[:, 1], p[:, 0]].double() for p in (a, b))
    ga, gb = (grad[p[:, 2], p[:, 1], p[:, 0]].double() for p in (a, b))
    t = ((va - iso) / (va - vb))[:, None]
    g = ga + t * (gb - ga)
    return (a.double() + t * unit[axis].double()) / cells, (-g if central else iso - g) / cells


def _functor_samples(size):
    """The demos' cubic and its gradient at texel centres, rounded to 32 bits after every operation."""
    x, y, z = (2.0 * ((torch.arange(n, device=DEV).float() + 0.5) / n) - 1.0 for n in size)
    x, y, z = x[None, None, :], y[None, :, None], z[:, None, None]
    v = 1.0 - 16.0 * x * y * z
    for c in (x, y, z):
        v = v - 4.0 * c * c
    return v, torch.stack(torch.broadcast_tensors(-16.0 * y * z - 8.0 * x, -16.0 * x * z - 8.0 * y,
                                                  -16.0 * x * y - 8.0 * z), 3)


def _reference_soup(case, seed):
    """(a, axis) of every vertex of the case, volume by volume."""
    if case["path"] == "batch":
        fields, isos = _batch_volumes(case, seed)
    elif case["path"] == "functor":
        fields, isos = [_functor_samples(_size(case))[0]], [_functor_iso(case, seed)]
    else:
        field, iso = _volume(case, seed)
        fields, isos = [field[..., 3] if field.dim() == 4 else field], [iso]
    return [_soup(_samples(case, f) < float(np.float32(iso))) for f, iso in zip(fields, isos)]


def _reference_vertices(case, seed):
    return sum(a.shape[0] for a, _ in _reference_soup(case, seed))


def _weld(case, a, axis):
    """Distinct edges, each vertex's edge, and the first vertex of each edge."""
    fx, fy, _ = _size(case)
    key = ((a[:, 2] * fy + a[:, 1]) * fx + a[:, 0]) * 3 + axis
    edge, back = torch.unique(key, return_inverse=True)
    first = torch.full((edge.numel(),), key.numel(), dtype=torch.int64, device=DEV)
    first.scatter_reduce_(0, back, torch.arange(key.numel(), device=DEV), "amin")
    return edge, back, first


def _reference_welded(case, seed):
    return _weld(case, *_reference_soup(case, seed)[0])[0].numel()


def _plain(case, field, iso, central):
    iso = float(np.float32(iso))
    f = _samples(case, field)
    a, axis = _soup(f < iso)
    return _geometry(f.double(), iso, a, axis, central), a, axis


def exact(case, seed):
    if _case_tables() is None:
        return None
    path, central = case["path"], case.get("normals") == "central"
    count = functools.partial(_reference_vertices, case)
    if path == "batch":
        parts = [_plain(case, f, iso, True)[0] for f, iso in zip(*_batch_volumes(case, seed))]
        p, n = (torch.cat([part[i] for part in parts]) for i in range(2))
        return _streams(p, n, _capacity(case, "vertices", count))
    if path == "functor":
        p, n = _gradient_mode(*_functor_samples(_size(case)), _functor_iso(case, seed), False)
        return {"feedback": _rows(torch.cat((n, p), 1), _capacity(case, "vertices", count))}
    field, iso = _volume(case, seed)
    if path == "autograd":
        a, axis = _soup(field < iso)
        f = field.double().requires_grad_(True)
        p, n = _geometry(f, iso, a, axis, central)
        w, u = (v[:, :3].double() for v in _cotangents(p.shape[0], seed))
        return {"grad": torch.autograd.grad([p, n], f, [w, u])[0]}
    if case["dtype"] == "f32x4":
        p, n = _gradient_mode(field[..., 3], field[..., :3], iso, central)
    else:
        (p, n), a, axis = _plain(case, field, iso, central)
    rows = _capacity(case, "vertices", count)
    if path != "indexed":
        return _streams(p, n, rows)
    edge, back, first = _weld(case, a, axis)
    first, order = torch.sort(first)
    out = _streams(p[first], n[first], _capacity(case, "welded", lambda seed: _reference_welded(case, seed)))
    return dict(out, indices=_rows(torch.argsort(order)[back], rows))


_WORK = {}


def work(case):
    """Field bytes read once and output bytes written once (a gradient's inputs
    and outputs too), for the vertices of seed 0; operations: a comparison per
    sample, and per vertex the crossing, the position and the normal."""
    if _key(case) not in _WORK:
        path = case["path"]
        n = _vertices(case, 0)
        if path == "batch":
            samples = sum(e ** 3 for e in _batch_sizes(case))
        else:
            samples = math.prod(_size(case))
        field_bytes = samples * {"f32": 4, "f32x4": 16, None: 0}.get(case.get("dtype"), 1)
        vertices = _welded(case, 0) if path == "indexed" else n
        out = {"functor": 24 * n, "indexed": 4 * n + 32 * vertices}.get(path, 32 * n)
        more = field_bytes if path == "autograd" else 0  # there `out` is the cotangents read, `more` the gradient written
        each = 40 * vertices * (2 if path == "autograd" else 1)
        _WORK[_key(case)] = {"bytes": field_bytes + out + more, "flops": samples * (13 if path == "functor" else 1) + each}
    return dict(_WORK[_key(case)])
