"""What a user of this codec has it do, as cases that can be timed: fields encoded to dataset
files, datasets opened, grids, boxes, coarse previews and batches of requests decoded, and the
differentiable decode trained through.

Sizes and tolerances are those of the repository's workloads (the 384x384x256 float64 field, the
1024^3 float32 field with fronts, uneven batches of axes 17-300, ROI serving with sides 32-512 and
downsampling 0-3, batches of 256^3 fields through the differentiable decode) and generic ones.
"""
from __future__ import annotations

import math
import os
import random
import tempfile

import numpy as np
import torch

import idx2_b200
from idx2_b200 import diff
from idx2_b200.synthetic import grf_field_torch

_TMP = "/dev/shm" if os.path.isdir("/dev/shm") else None


def listed():
    return [
        # one small 2D slice from host memory to files: the smallest call, all latency
        {"name": "encode_slice", "kind": "encode", "dims": "200x150x1", "dtype": "float64", "levels": 1,
         "tol": 1e-4, "field": "grf", "where": "host"},
        # a smooth simulation variable of double precision, in situ (the field is on the GPU)
        {"name": "encode_f64_384", "kind": "encode", "dims": "384x384x256", "dtype": "float64", "levels": 2,
         "tol": 1e-3, "field": "bumps", "where": "cuda"},
        # the large single field: turbulence with sharp fronts
        {"name": "encode_f32_1024", "kind": "encode", "dims": "1024x1024x1024", "dtype": "float32", "levels": 3,
         "tol": 1e-3, "field": "fronts", "where": "cuda"},
        # many variables of uneven sizes, types and levels at once, some of them 2D
        {"name": "encode_batch_16", "kind": "encode_batch", "fields": 16, "lo": 33, "hi": 300, "tol": 1e-3,
         "shapes": 1},
        # a small box of a resident dataset at full resolution: an interactive probe
        {"name": "decode_box", "kind": "decode", "dims": "256x256x256", "dtype": "float32", "levels": 2,
         "tol": 1e-5, "field": "grf", "box": "96x80x64", "ds": 0, "at": 1e-5},
        # the whole double-precision field read back on the GPU
        {"name": "decode_f64_384", "kind": "decode", "dims": "384x384x256", "dtype": "float64", "levels": 2,
         "tol": 1e-3, "field": "bumps", "box": "", "ds": 0, "at": 1e-3},
        # the whole large field read back on the GPU
        {"name": "decode_f32_1024", "kind": "decode", "dims": "1024x1024x1024", "dtype": "float32", "levels": 3,
         "tol": 1e-3, "field": "fronts", "box": "", "ds": 0, "at": 1e-3},
        # a preview: half resolution per axis, a coarser tolerance than the dataset holds
        {"name": "decode_coarse_512", "kind": "decode", "dims": "512x512x512", "dtype": "float32", "levels": 3,
         "tol": 1e-5, "field": "grf", "box": "", "ds": 1, "at": 1e-2},
        # one serving batch: boxes of sides 32-512, downsampling 0-3 per axis, tolerances 1e-6..1e-1
        {"name": "serve_24", "kind": "decode_batch", "dims": "1024x512x512", "dtype": "float32", "levels": 3,
         "tol": 1e-6, "requests": 24, "lo": 32, "hi": 512, "shapes": 2},
        # a dataset on disk into a host array: open, decode, close
        {"name": "load_f32_odd", "kind": "load", "dims": "301x203x157", "dtype": "float32", "levels": 2,
         "tol": 1e-4, "field": "grf"},
        # a training step's decode, forward and backward
        {"name": "diff_f32_32x256", "kind": "diff", "dims": "256x256x256", "dtype": "float32", "levels": 2,
         "tol": 1e-4, "batch": 32},
        # the same in double precision on one odd field
        {"name": "diff_f64_odd", "kind": "diff", "dims": "131x97x70", "dtype": "float64", "levels": 2,
         "tol": 1e-4, "batch": 1},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _levels_for(dims, most):
    """As many levels as the format's rules take for these sizes, at most `most`."""
    n = most
    while n > 1 and idx2_b200.check_params(_params(dims, "float32", n, 1e-3)) != 0:
        n -= 1
    return n


def draw(rng):
    kind = rng.choice(["encode", "encode", "encode_batch", "decode", "decode", "decode_batch", "load", "diff"])
    dtype = rng.choice(["float32", "float64"])
    if kind == "encode_batch":
        return {"kind": kind, "fields": rng.randint(2, 16), "lo": 33, "hi": rng.randint(64, 300),
                "tol": _log_uniform(rng, 1e-5, 1e-2), "shapes": rng.randrange(1 << 20)}
    if kind == "diff":
        side = _log_uniform(rng, 40, 256)
        dims = [max(33, int(side * rng.uniform(0.6, 1.0))) for _ in range(3)]
        most = 32 * 256 ** 3 if dtype == "float32" else 32 * 128 ** 3
        batch = int(_log_uniform(rng, 1, max(1.0, min(32.0, 0.9 * most / (dims[0] * dims[1] * dims[2])))))
        return {"kind": kind, "dims": "%dx%dx%d" % tuple(dims), "dtype": dtype, "levels": _levels_for(dims, 2),
                "tol": _log_uniform(rng, 1e-6, 1e-3), "batch": max(1, batch)}
    top = {"encode": 640, "decode": 640, "decode_batch": 640, "load": 320}[kind]
    side = _log_uniform(rng, 256 if kind == "decode_batch" else 64, top)
    dims = [max(33, int(side * rng.uniform(0.6, 1.0))) for _ in range(3)]
    if rng.random() < 0.15 and kind in ("encode", "decode"):
        dims[2] = 1
    levels = _levels_for(dims, rng.randint(1, 3))
    tol = _log_uniform(rng, 1e-6, 1e-2)
    text = "%dx%dx%d" % tuple(dims)
    if kind == "encode":
        return {"kind": kind, "dims": text, "dtype": dtype, "levels": levels, "tol": tol, "field": "grf",
                "where": rng.choice(["host", "cuda", "cuda"])}
    if kind == "decode":
        box = ""
        if rng.random() < 0.5:
            box = "%dx%dx%d" % tuple(max(1, min(d, int(d * rng.uniform(0.1, 0.9)))) for d in dims)
        return {"kind": kind, "dims": text, "dtype": dtype, "levels": levels, "tol": tol, "field": "grf", "box": box,
                "ds": rng.choice([0, 0, 1, 2]), "at": _log_uniform(rng, tol, max(tol * 1.01, 1e-1))}
    if kind == "decode_batch":
        return {"kind": kind, "dims": text, "dtype": dtype, "levels": levels, "tol": tol,
                "requests": int(_log_uniform(rng, 2, 24)), "lo": 32, "hi": rng.randint(64, 512),
                "shapes": rng.randrange(1 << 20)}
    return {"kind": kind, "dims": text, "dtype": dtype, "levels": levels, "tol": tol, "field": "grf"}


def _dims(case):
    return tuple(int(v) for v in case["dims"].split("x"))


def _params(dims, dtype, levels, tol):
    return idx2_b200.Params(dims=dims, dtype=dtype, brick_dims=(32, 32, 1) if dims[2] == 1 else (32, 32, 32),
                            num_levels=levels, tolerance=tol)


def _bumps(dims, seed):
    """Sum of Gaussian bumps, low-wavenumber waves and weak noise, float64 (nz, ny, nx)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n = 64
    ax = [torch.arange(d, device="cuda", dtype=torch.float64) for d in dims]
    centre = [torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * d for d in dims]
    sigma = 8 + 32 * torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    amp = torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
    ex, ey, ez = [torch.exp(-(a[None, :] - c[:, None]) ** 2 / (2 * sigma[:, None] ** 2)) for a, c in zip(ax, centre)]
    zy = ((amp[:, None] * ez)[:, :, None] * ey[:, None, :]).reshape(n, -1)
    f = (zy.T @ ex).reshape(dims[2], dims[1], dims[0])
    for k in range(1, 5):
        wx, wy, wz = [2 * math.pi * k * a / max(d, 1) for a, d in zip(ax, dims)]
        f += (0.5 / k) * torch.cos(wy)[None, :, None] * torch.sin(wx)[None, None, :] * \
            torch.sin(wz + 0.3 * k)[:, None, None]
    f += 1e-4 * torch.randn(f.shape, generator=gen, device="cuda", dtype=torch.float64)
    return f


def _field(dims, dtype, kind, seed):
    """A field on the GPU, (nz, ny, nx)."""
    if kind == "bumps":
        f = _bumps(dims, seed)
    else:
        f = grf_field_torch(dims[0], dims[1], dims[2], seed=seed, scale="unit",
                            n_fronts=20 if kind == "fronts" else 0, device="cuda")
    return f.to(torch.float32 if dtype == "float32" else torch.float64).contiguous()


class _Folder:
    """A folder in memory that goes with its state."""

    def __init__(self):
        self._dir = tempfile.TemporaryDirectory(prefix="idx2_cases_", dir=_TMP, ignore_cleanup_errors=True)
        self.path = self._dir.name


def _files(path, dims, size, tol):
    """The bytes of a dataset's files in the order of their names, mapped. A field of other values
    compresses to other sizes: each file is given the length that its level may have at most (a
    hole past its end, read as zeros; the next encode cuts it off), so that arrays of one case
    have one shape."""
    n = dims[0] * dims[1] * dims[2]
    got = []
    for where, folders, names in os.walk(path):
        folders.sort()
        for name in sorted(names):
            p = os.path.join(where, name)
            level = int(name[1:3]) if name.endswith(".bin") else None
            most = 1 << 16
            if level is not None:
                most += int(min(1.25 * n * size, max(1 << 26, 1.5 * _stream_bytes(n, tol)))) >> level
            if os.path.getsize(p) > most:
                raise RuntimeError("%s is larger than its level may be" % p)
            os.truncate(p, most)
            got.append(np.memmap(p, dtype=np.uint8, mode="r"))
    return got


def _dataset_files(case, seed):
    d = _Folder()
    f = _field(_dims(case), case["dtype"], case.get("field", "grf"), seed)
    idx2_b200.encode(f, out_dir=d.path, name="data", field_name="f", num_levels=case["levels"], tolerance=case["tol"])
    return d, os.path.join(d.path, "data", "f.idx2")


def _out_shape(first, last, ds):
    """The output grid of a box: first sample rounded down, last rounded up to the stride."""
    n = []
    for f, l, k in zip(first, last, ds):
        s = 1 << k
        n.append(((-(-l // s)) * s - (f // s) * s) // s + 1)
    return n


def _place(place, dims, side, offset):
    """First sample of a box: `offset` past a multiple of 8 on each axis, which keeps the size of
    the output grid (downsampling is at most 3) the same wherever the box lies."""
    return [o + 8 * place.randint(0, (d - n - o) // 8) for d, n, o in zip(dims, side, offset)]


def _requests(case, seed):
    """The batch's boxes: their shapes, strides and tolerances are the case's, their places the seed's."""
    shape, place = random.Random(case["shapes"]), random.Random(seed)
    dims = _dims(case)
    got = []
    for _ in range(case["requests"]):
        side = [min(shape.randint(case["lo"], case["hi"]), d) for d in dims]
        first = _place(place, dims, side, [shape.randint(0, min(7, d - n)) for d, n in zip(dims, side)])
        ds = [shape.randint(0, 3) for _ in dims]
        got.append({"first": first, "last": [f + s - 1 for f, s in zip(first, side)], "downsampling": ds,
                    "tolerance": _log_uniform(shape, case["tol"], max(1e-1, case["tol"]))})
    return got


def _batch_fields(case):
    """(dims, dtype, levels) of the uneven batch."""
    shape = random.Random(case["shapes"])
    got = []
    for i in range(case["fields"]):
        dims = [shape.randint(case["lo"], case["hi"]) for _ in range(3)]
        if shape.randrange(8) == 0:
            dims[2] = 1
        got.append((tuple(dims), "float32" if i % 2 == 0 else "float64", _levels_for(dims, shape.randint(1, 3))))
    return got


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "encode":
        f = _field(_dims(case), case["dtype"], case["field"], seed)
        s["field"] = f.cpu().numpy() if case["where"] == "host" else f
        s["dir"] = _Folder()
    elif kind == "encode_batch":
        fields = _batch_fields(case)
        s["fields"] = [_field(d, t, "grf", seed * 1000 + i) for i, (d, t, _) in enumerate(fields)]
        s["names"] = ["v%02d" % i for i in range(len(fields))]
        s["levels"] = [n for _, _, n in fields]
        s["tols"] = [case["tol"]] * len(fields)
        s["dir"] = _Folder()
    elif kind == "decode":
        folder, path = _dataset_files(case, seed)
        s["ds"] = idx2_b200.Dataset(path)
        dims, k = _dims(case), case["ds"]
        ds = tuple(k if d > 1 else 0 for d in dims)
        first, last = None, None
        if case["box"]:
            place = random.Random(seed)
            side = [int(v) for v in case["box"].split("x")]
            first = _place(place, dims, side, [min(3, d - n) for d, n in zip(dims, side)])
            last = [f + n - 1 for f, n in zip(first, side)]
        s["request"] = {"first": first, "last": last, "downsampling": ds, "tolerance": case["at"]}
        _, n, _ = s["ds"].output_grid(first, last, ds)
        s["out"] = torch.zeros((n[2], n[1], n[0]), device="cuda",
                               dtype=torch.float32 if case["dtype"] == "float32" else torch.float64)
    elif kind == "decode_batch":
        folder, path = _dataset_files(case, seed)
        s["ds"] = idx2_b200.Dataset(path)
        s["requests"] = _requests(case, seed)
    elif kind == "load":
        s["dir"], s["path"] = _dataset_files(case, seed)
    else:
        fmt = diff.Format(_dims(case), case["dtype"], case["levels"])
        got = []
        for i in range(case["batch"]):
            folder, path = _dataset_files(case, seed * 1000 + i)
            ds = idx2_b200.Dataset(path)
            got.append(diff.coefficients(ds, fmt, case["tol"]))
            ds.close()
        s["fmt"] = fmt
        s["coeffs"] = torch.stack(got).requires_grad_(True)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        s["grad"] = torch.randn((case["batch"],) + fmt.shape, generator=gen, device="cuda", dtype=s["coeffs"].dtype)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "encode":
        idx2_b200.encode(state["field"], out_dir=state["dir"].path, name="data", field_name="f",
                         num_levels=case["levels"], tolerance=case["tol"])
        return _files(state["dir"].path, _dims(case), 4 if case["dtype"] == "float32" else 8, case["tol"])
    if kind == "encode_batch":
        idx2_b200.encode_batch(state["fields"], out_dir=state["dir"].path, names=state["names"],
                               num_levels=state["levels"], tolerances=state["tols"])
        return [_files(os.path.join(state["dir"].path, name), d, 4 if t == "float32" else 8, case["tol"])
                for name, (d, t, _) in zip(state["names"], _batch_fields(case))]
    if kind == "decode":
        return state["ds"].decode(out=state["out"], **state["request"])
    if kind == "decode_batch":
        return state["ds"].decode_batch(state["requests"], device_out=True)
    if kind == "load":
        ds = idx2_b200.Dataset(state["path"])
        grid = ds.decode(tolerance=case["tol"])
        ds.close()
        return grid
    grid = diff.decode_diff(state["coeffs"], state["fmt"])
    (g,) = torch.autograd.grad(grid, state["coeffs"], state["grad"])
    return {"grid": grid.detach(), "grad": g}


def _stream_bytes(samples, tol):
    """Compressed size: these fields take about log2(1 / tolerance) bits a sample (1.25 GB for
    1024^3 at 1e-3, 11 GB for 4.3 G samples at 1e-6)."""
    return samples * max(1.0, math.log2(1.0 / tol)) / 8


def work(case):
    kind = case["kind"]
    size = 4 if case.get("dtype") == "float32" else 8
    if kind == "encode_batch":
        raw = comp = 0.0
        for d, t, _ in _batch_fields(case):
            n = d[0] * d[1] * d[2]
            raw += n * (4 if t == "float32" else 8)
            comp += _stream_bytes(n, case["tol"])
        return {"bytes": raw + comp, "flops": 0.0}
    dims = _dims(case)
    n = dims[0] * dims[1] * dims[2]
    if kind in ("encode", "load"):
        smooth = 16.0 if case["field"] == "bumps" else 1.0  # the smooth field compresses much further
        return {"bytes": n * size + _stream_bytes(n, case["tol"]) / smooth, "flops": 0.0}
    if kind == "diff":
        levels, c, nb = case["levels"], 0, [-(-d // 32) for d in dims]
        for _ in range(levels):
            c += nb[0] * nb[1] * nb[2] * 33 ** 3
            nb = [-(-b // 2) for b in nb]
        # forward: coefficients to grid; backward: its gradient to theirs
        return {"bytes": 2.0 * case["batch"] * (n + c) * size, "flops": 0.0}
    boxes = _requests(case, 0) if kind == "decode_batch" else [
        {"first": [0, 0, 0], "last": [int(v) - 1 for v in (case["box"] or case["dims"]).split("x")],
         "downsampling": [case["ds"] if d > 1 else 0 for d in dims], "tolerance": case["at"]}]
    total = 0.0
    for b in boxes:
        m = float(np.prod(_out_shape(b["first"], b["last"], b["downsampling"])))
        smooth = 16.0 if case.get("field") == "bumps" else 1.0
        total += m * size + _stream_bytes(m, max(b["tolerance"], case["tol"])) / smooth
    return {"bytes": total, "flops": 0.0}


# ---------------------------------------------------------------------------
# The differentiable decode in 64 bits: the inverse zfp and CDF5/3 lines as matrices made from
# their steps, the subband weights, the low band handed from parent to child.
# ---------------------------------------------------------------------------

def _zfp_line(v):
    x, y, z, w = v
    y += w * 0.5
    w -= y * 0.5
    y += w
    w = 2 * w - y
    z += x
    x = 2 * x - z
    y += z
    z = 2 * z - y
    w += x
    x = 2 * x - w
    return [x, y, z, w]


def _cdf_line(v):
    v = list(v)
    for x in range(1, 33, 2):
        q = v[x] * 0.25
        v[x - 1] -= q
        v[x + 1] -= q
    for x in range(1, 33, 2):
        v[x] += (v[x - 1] + v[x + 1]) * 0.5
    return v


def _matrix(line, n):
    return torch.tensor(np.array([line([float(i == j) for i in range(n)]) for j in range(n)]).T, device="cuda",
                        dtype=torch.float64)


def _along(t, axis, m):
    return torch.movedim(torch.movedim(t, axis, -1) @ m.T, -1, axis)


def _exact_grid(c, dims, levels):
    """One field's grid from its coefficients, both float64; autograd gives the adjoint."""
    m4, m33 = _matrix(_zfp_line, 4), _matrix(_cdf_line, 33)
    zfp = {n: torch.block_diag(*([m4] * 4 + [torch.ones(1, 1, device="cuda", dtype=torch.float64)] * (n - 16)))
           for n in (16, 17)}
    scal = [math.sqrt((3 * 4 ** i - (4 ** i - 1) / 3) / 2 ** (i + 1)) for i in range(levels)]
    wave = [math.sqrt((23 * 4 ** i - 33 * (4 ** i - 1) / 3) / 2 ** (i + 5)) for i in range(levels)]
    grids, base = [], 0
    nb = [-(-d // 32) for d in dims]
    for _ in range(levels):
        n = nb[0] * nb[1] * nb[2] * 33 ** 3
        grids.append((tuple(nb), base, base + n))
        base += n
        nb = [-(-b // 2) for b in nb]
    prev = None
    for lv in range(levels - 1, -1, -1):
        (bx, by, bz), b0, b1 = grids[lv]
        co = c[b0:b1].reshape(bz, by, bx, 33, 33, 33)
        f = torch.zeros_like(co)
        for hz in (0, 1):
            for hy in (0, 1):
                for hx in (0, 1):
                    s = co[..., hz::2, hy::2, hx::2]
                    for axis in (3, 4, 5):
                        s = _along(s, axis, zfp[s.shape[axis]])
                    if hx or hy or hz or lv == levels - 1:
                        s = s / math.prod(wave[lv] if h else scal[lv] for h in (hx, hy, hz))
                    f[..., hz::2, hy::2, hx::2] = s
        if prev is not None:
            pz, py, px = prev.shape[:3]
            low = prev[..., :32, :32, :32].reshape(pz, py, px, 2, 16, 2, 16, 2, 16)
            low = low.permute(0, 3, 1, 5, 2, 7, 4, 6, 8).reshape(2 * pz, 2 * py, 2 * px, 16, 16, 16)
            f[..., 0:32:2, 0:32:2, 0:32:2] = low[:bz, :by, :bx]
        for axis in (3, 4, 5):
            f = _along(f, axis, m33)
        prev = f
    bz, by, bx = prev.shape[:3]
    grid = prev[..., :32, :32, :32].permute(0, 3, 1, 4, 2, 5).reshape(32 * bz, 32 * by, 32 * bx)
    return grid[:dims[2], :dims[1], :dims[0]]


def exact(case, seed):
    """The differentiable decode in 64 bits. The other cases have none: an encode's output is
    bytes, and a decode's is what the format's integer arithmetic says, bit for bit."""
    if case["kind"] != "diff":
        return None
    s = prepare(case, seed)
    grid, grad = [], []
    for i in range(case["batch"]):
        c = s["coeffs"][i].detach().double().requires_grad_(True)
        g = _exact_grid(c, _dims(case), case["levels"])
        (d,) = torch.autograd.grad(g, c, s["grad"][i].double())
        grid.append(g.detach())
        grad.append(d)
    return {"grid": torch.stack(grid), "grad": torch.stack(grad)}
