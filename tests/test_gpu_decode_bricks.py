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
