"""The value range of a field whose least or greatest sample is a zero, and which holds zeros of
both signs: the sign in the metadata is that of the first zero in the reference's order (bricks in
encode order, x fastest inside a brick), whatever the kernel. Files byte for byte against the
oracle's coder."""
import numpy as np
import pytest

from idx2_files import compare_dirs
from oracle_tools import oracle_encode


def _zeros_of_both_signs(dims, dtype, seed, negative):
    rng = np.random.default_rng(seed)
    f = np.abs(rng.standard_normal(dims[::-1])) + 0.1
    f[rng.random(f.shape) < 0.02] = 0.0
    f[:, : dims[1] // 3, : dims[0] // 2] += 0.5  # (the first zero is not the first brick's first sample)
    sign = np.where(rng.random(f.shape) < 0.5, -1.0, 1.0)
    f = np.where(f == 0, f * sign, -f if negative else f)
    return np.ascontiguousarray(f.astype(dtype))


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(64, 64, 64), (61, 33, 40), (97, 64, 33), (90, 70, 1)])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_zero_extremum_has_the_first_zeros_sign(idx2g, tmp_path, dims, dtype):
    brick = (32, 32, 1) if dims[2] == 1 else (32, 32, 32)
    for seed in range(3):
        for negative in (False, True):
            f = _zeros_of_both_signs(dims, dtype, seed, negative)
            d = tmp_path / f"{seed}{negative}"
            d.mkdir()
            f.tofile(str(d / "in.raw"))
            rc, err = oracle_encode(str(d / "in.raw"), dims, dtype, 1, 1e-3, str(d / "o"), brick=brick)
            assert rc == 0, err
            idx2g.encode(f, out_dir=str(d / "g"), name="kat", field_name="f", num_levels=1, tolerance=1e-3,
                         brick_dims=brick)
            assert compare_dirs(str(d / "o" / "kat"), str(d / "g" / "kat")) == [], (seed, negative)
            # a batch of two: the fields share launches, and a sign each
            idx2g.encode_batch([f, f[::-1].copy()], out_dir=str(d / "b"), names=["kat", "rev"], field_names=["f", "f"],
                               num_levels=[1, 1], tolerances=[1e-3, 1e-3])
            got = (d / "b" / "kat" / "f.idx2").read_text().split("min-max")[1].split(")")[0]
            assert got == (d / "o" / "kat" / "f.idx2").read_text().split("min-max")[1].split(")")[0]
