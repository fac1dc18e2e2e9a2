"""Fields of values far apart and of values that are no numbers: what the coder cannot hold is
refused with an error, and what it can hold gives the files of the oracle's coder."""
import numpy as np
import pytest

from idx2_files import compare_dirs
from oracle_tools import oracle_encode

DIMS = (64, 64, 64)


def _base():
    return np.random.default_rng(11).standard_normal(DIMS[::-1])


@pytest.mark.gpu
@pytest.mark.parametrize("big,tol", [(9e37, 1e-2), (2e37, 1e-7)])
def test_blocks_too_far_apart_are_refused(idx2g, tmp_path, big, tol):
    """Samples near the largest float32: blocks whose transformed samples no longer fit the type have
    exponent 0, the others some 125, so that a subband spans 141 or 158 channel keys, more than the 128
    there is room for: an error, from one encode and from a batch, and the context encodes on."""
    f = _base().astype("float32")
    far = (np.sign(f) * np.float32(big)).astype("float32")
    for _ in range(2):
        with pytest.raises(idx2g.Idx2Error, match="DeviceStreamOverflow"):
            idx2g.encode(far, out_dir=str(tmp_path), name="far", field_name="f", num_levels=1, tolerance=tol)
    with pytest.raises(idx2g.Idx2Error, match="DeviceStreamOverflow"):
        idx2g.encode_batch([f, far], out_dir=str(tmp_path), names=["a", "far"], field_names=["f", "f"],
                           num_levels=[1, 1], tolerances=[tol, tol])
    f.tofile(str(tmp_path / "in.raw"))
    assert oracle_encode(str(tmp_path / "in.raw"), DIMS, "float32", 1, tol, str(tmp_path / "o"))[0] == 0
    idx2g.encode(f, out_dir=str(tmp_path / "g"), name="kat", field_name="f", num_levels=1, tolerance=tol)
    assert compare_dirs(str(tmp_path / "o" / "kat"), str(tmp_path / "g" / "kat")) == []


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf], ids=str)
@pytest.mark.parametrize("share", [0.0, 0.01])
def test_values_that_are_no_numbers_match_oracle(idx2g, tmp_path, dtype, value, share):
    """One such value (share 0), or some in every brick: they spread over their bricks."""
    f = _base()
    f[np.random.default_rng(5).random(f.shape) < share] = value
    f[0, 7, 9] = value
    f = f.astype(dtype)
    for tol in (1e-2, 1e-6):
        d = tmp_path / str(tol)
        d.mkdir()
        f.tofile(str(d / "in.raw"))
        assert oracle_encode(str(d / "in.raw"), DIMS, dtype, 1, tol, str(d / "o"))[0] == 0
        idx2g.encode(f, out_dir=str(d / "g"), name="kat", field_name="f", num_levels=1, tolerance=tol)
        assert compare_dirs(str(d / "o" / "kat"), str(d / "g" / "kat")) == [], tol


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-3, 1e100, 1e300])
def test_bricks_far_apart_match_oracle(idx2g, tmp_path, scale):
    """Bricks whose exponents lie up to 1,000 apart: from 256 channel keys in a chunk on, more than the
    device packer's window, the host packs."""
    f = _base()
    f[:32, :32, :32] *= scale
    f[32:, 32:, 32:] *= scale ** 0.5
    f.tofile(str(tmp_path / "in.raw"))
    assert oracle_encode(str(tmp_path / "in.raw"), DIMS, "float64", 1, 1e-3, str(tmp_path / "o"))[0] == 0
    for i in range(3):
        idx2g.encode(f, out_dir=str(tmp_path / f"g{i}"), name="kat", field_name="f", num_levels=1, tolerance=1e-3)
        assert compare_dirs(str(tmp_path / "o" / "kat"), str(tmp_path / f"g{i}" / "kat")) == []
