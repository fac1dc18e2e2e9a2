"""Pageable host arrays at the sizes where a copy changes its form (4 MB, pieces of 1 MB, ragged
ends): a decode into a numpy array equals the decode on the device, and an encode of a numpy
array writes the files of the encode of the same CUDA tensor."""
import pytest

DIMS = [(128, 128, 63), (128, 128, 64), (129, 131, 67), (200, 150, 101)]


@pytest.mark.gpu
@pytest.mark.parametrize("dims", DIMS)
def test_pageable_arrays_match_device_ones(idx2g, tmp_path, dims):
    import torch
    from idx2_b200.synthetic import grf_field_torch
    f = grf_field_torch(*dims, seed=9, device="cuda")
    host = f.cpu().numpy()
    for name, field in (("d", f), ("h", host)):
        idx2g.encode(field, out_dir=str(tmp_path / name), name="t", field_name="f", num_levels=1, tolerance=1e-4)
    files = [{p.relative_to(tmp_path / n): p.read_bytes() for p in (tmp_path / n).rglob("*") if p.is_file()}
             for n in ("d", "h")]
    assert files[0] == files[1] and files[0]
    ds = idx2g.Dataset(str(tmp_path / "h" / "t" / "f.idx2"))
    out = torch.empty(f.shape, device="cuda")
    ds.decode(out=out)
    assert ds.decode().tobytes() == out.cpu().numpy().tobytes()
    ds.close()
