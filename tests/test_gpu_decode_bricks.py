"""The lane-per-block decode of 3D bricks (k_decode_bricks) against the general single-kernel
wavefront, which idx2g_decode_noalloc runs, bit for bit: every range of planes per block that
takes a form of its own (up to 16, up to 26, up to 44, more), both dtypes, odd sizes, boxes,
strides that skip blocks, and output rows that can and cannot leave as 16-byte stores."""
import pytest

from test_zz_no_alloc import _noalloc

DIMS = (101, 70, 66)  # 4 x 3 x 3 bricks on level 0, 2 x 2 x 2 on level 1

REQUESTS = [
    {"ds": (0, 0, 0)},
    {"ds": (1, 0, 2)},
    {"ds": (2, 2, 2)},
    {"ds": (0, 0, 0), "first": (31, 32, 5), "last": (66, 69, 40)},
    {"ds": (0, 1, 0), "first": (5, 3, 1), "last": (38, 33, 32)},
]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [("float32", 1e-1), ("float32", 1e-3), ("float32", 1e-6), ("float32", 1e-9),
                                       ("float64", 1e-2), ("float64", 1e-8), ("float64", 1e-11),
                                       ("float64", 1e-14)])
def test_brick_decode_matches_wavefront(idx2g, tmp_path, dtype, tol):
    import numpy as np
    import torch
    from idx2_b200.synthetic import grf_field
    f = grf_field(*DIMS, seed=5, scale="unit", n_fronts=1).astype(dtype)
    f[:, :20, :40] = np.float32(0.25)  # blocks without planes beside full ones
    idx2g.encode(f, out_dir=str(tmp_path), name="b", field_name="f", num_levels=2, tolerance=tol)
    ds = idx2g.Dataset(str(tmp_path / "b" / "f.idx2"))
    dt = torch.float32 if dtype == "float32" else torch.float64
    for req in REQUESTS:
        for at in (0.0, 30 * tol):
            r = dict(req, tol=at)
            _, dims, _ = ds.output_grid(r.get("first"), r.get("last"), r["ds"])
            shape = (dims[2], dims[1], dims[0])
            ours = torch.empty(shape, dtype=dt, device="cuda")
            want = torch.empty(shape, dtype=dt, device="cuda")
            ds.decode(first=r.get("first"), last=r.get("last"), downsampling=r["ds"], tolerance=at, out=ours)
            assert _noalloc(idx2g, ds, r, want) == 0
            torch.cuda.synchronize()
            assert ours.cpu().numpy().tobytes() == want.cpu().numpy().tobytes(), r
    ds.close()


@pytest.fixture(scope="module")
def many_bricks(idx2g, tmp_path_factory):
    """Fields of one level and 700 bricks: 8 warps per brick, as in every launch of more bricks than
    SMs, and on the whole grid two (brick, subband) units per warp of the plane kernel (5,600 units).
    A third of the field is smooth, a third noisy, and a slab constant, so that units that share a warp
    differ in channels and length."""
    import numpy as np
    from idx2_b200.synthetic import grf_field
    d = tmp_path_factory.mktemp("many")
    f = grf_field(320, 320, 200, seed=6, scale="unit")
    x = np.arange(320) // 7 % 3
    f = np.where(x == 0, np.linspace(0, 1, 320), np.where(x == 1, f, 0.1 * f * f))
    f[:, 40:90, :] = 0.5
    f[:, :, 96:128] *= 1e-3
    got = {}
    for dtype, tol in (("float32", 1e-4), ("float64", 1e-8)):
        idx2g.encode(f.astype(dtype), out_dir=str(d / dtype), name="b", field_name="f", num_levels=1, tolerance=tol)
        got[dtype] = idx2g.Dataset(str(d / dtype / "b" / "f.idx2"))
    yield got
    for ds in got.values():
        ds.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("req", [
    {"ds": (0, 0, 0)},                                                      # rows of 16-byte stores
    {"ds": (0, 1, 0)},                                                      # the same, every other row
    {"ds": (0, 0, 1)},
    {"ds": (1, 0, 0)},                                                      # rows of single stores
    {"ds": (0, 0, 0), "first": (32, 5, 3), "last": (287, 300, 190)},        # 16-byte stores from a brick's edge on
    {"ds": (0, 0, 0), "first": (30, 0, 0), "last": (285, 319, 199)},        # whole bricks, not at 16 bytes
], ids=str)
def test_many_bricks_match_wavefront(idx2g, many_bricks, dtype, req):
    """Launches of more bricks than SMs (8 warps each), units in pairs, and float rows that leave as
    16-byte stores, at unit and other strides, against the wavefront kernel."""
    import torch
    ds = many_bricks[dtype]
    for at in (0.0, 1e-2):
        r = dict(req, tol=at)
        _, dims, _ = ds.output_grid(r.get("first"), r.get("last"), r["ds"])
        ours, want = (torch.empty((dims[2], dims[1], dims[0]), dtype=getattr(torch, dtype), device="cuda")
                      for _ in range(2))
        ds.decode(first=r.get("first"), last=r.get("last"), downsampling=r["ds"], tolerance=at, out=ours)
        assert _noalloc(idx2g, ds, r, want) == 0
        torch.cuda.synchronize()
        assert torch.equal(ours.view(torch.uint8), want.view(torch.uint8)), at


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_large_decode_equals_its_boxes(idx2g, tmp_path, dtype):
    """Two levels, 196 bricks on the coarser one (kept by launches of 8 warps per brick): the whole grid
    against small boxes of it, whose bricks take 16 warps (test_brick_decode_matches_wavefront)."""
    import torch
    from idx2_b200.synthetic import grf_field_torch
    f = grf_field_torch(448, 448, 256, seed=8, device="cuda").to(getattr(torch, dtype))
    idx2g.encode(f, out_dir=str(tmp_path), name="b", field_name="f", num_levels=2, tolerance=1e-4)
    ds = idx2g.Dataset(str(tmp_path / "b" / "f.idx2"))
    whole = torch.empty_like(f)
    ds.decode(out=whole)
    for first in ((0, 0, 0), (30, 200, 100), (383, 383, 191), (224, 64, 31)):
        last = [a + 64 for a in first]
        box = torch.empty((65, 65, 65), dtype=f.dtype, device="cuda")
        ds.decode(first=first, last=last, out=box)
        x, y, z = first
        want = whole[z:z + 65, y:y + 65, x:x + 65].contiguous()
        assert torch.equal(box.view(torch.uint8), want.view(torch.uint8)), first
    ds.close()
