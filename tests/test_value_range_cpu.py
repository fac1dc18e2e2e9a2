"""The value range in the metadata file, written with 20 decimals as the reference does
(Core/idx2Common.cpp:150): values of any size, up to 310 digits before the point."""
import re

import numpy as np
import pytest

from oracle_tools import oracle_encode


@pytest.mark.parametrize("least,greatest", [(-1.5, 2.25), (-1e200, 1e300), (-3e299, 4e298)])
def test_min_max_of_any_size(tmp_path, least, greatest):
    f = np.zeros((64, 64, 64))
    f[0, 0, 0], f[63, 63, 63] = least, greatest
    f.tofile(str(tmp_path / "in.raw"))
    assert oracle_encode(str(tmp_path / "in.raw"), (64, 64, 64), "float64", 1, 1e-3, str(tmp_path / "o"))[0] == 0
    text = (tmp_path / "o" / "kat" / "f.idx2").read_text(errors="replace").split("\n\n-----")[0]
    m = re.search(r"\(min-max (\S+) (\S+)\)\n    \(accuracy", text)
    assert m and (float(m[1]), float(m[2])) == (least, greatest)
    assert text.count("(") == text.count(")")
