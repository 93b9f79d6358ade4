"""Error of the FP64 passes' table-driven log2 against 80-bit log2
(csrc/kernels.cuh, csrc/log2_table.cuh).

Bars, from the roundings there are.  The table's values are doubles to 2^-13 of
their last place (at most 2^-53 each): 2^-66.  The polynomial's own error is 9e-19
< 2^-59.9, its rounding at most a few 2^-53 of |r q| <= 2^-8.4: 2^-60.  The sum of
exponent and table value rounds once and the last fma once, half an ulp of a number
of at most the result's size plus 2^-8:
  * |x - 1| <= 2^-7: that sum is exact there and the result below 0.0114, half an
    ulp of it 2^-60: 2^-58 together;
  * 2^-30 <= x <= 16: an ulp of max(1, |result|) and 2^-58."""
import os
import re

import numpy as np
import pytest

from conftest import REPO

ROW = re.compile(r"\{(-?0x[0-9a-fp.+-]+), (-?0x[0-9a-fp.+-]+)\}")


def test_rows():
    """-log2 c is the nearest double to what it stands for, c next to 1 / F."""
    text = open(os.path.join(REPO, "flexmm_b200", "csrc", "log2_table.cuh")).read()
    rows = np.array([[float.fromhex(v) for v in r] for r in ROW.findall(text)])
    assert rows.shape == (257, 2) and tuple(rows[0]) == (1.0, 0.0) and tuple(rows[256]) == (0.5, 1.0)
    c, v = rows.T
    assert np.max(np.abs(c * (1 + np.arange(257) / 256) - 1)) < 2e-11
    exact = -np.log2(c.astype(np.longdouble))
    # 80-bit logarithms are good to about 2^-64 here: the rows' 2^-13 of an ulp at most
    # 2^-66; what is left of the nearest-double distance is within 2^-62
    assert np.max(np.abs(np.asarray(exact - v, dtype=np.float64))) < 2.0 ** -62


def _error(x):
    from test_gpu_log2 import _run
    got, _ = _run(x)
    exact = np.log2(x.astype(np.longdouble))
    assert np.finfo(np.longdouble).eps < 1e-18
    return np.asarray(got - exact, dtype=np.float64), np.asarray(exact, dtype=np.float64)


@pytest.mark.gpu
def test_error_next_to_one(built_lib):
    rng = np.random.default_rng(3)
    e, _ = _error(1.0 + rng.uniform(-2.0 ** -7, 2.0 ** -7, 400_000))
    assert np.abs(e).max() <= 2.0 ** -58


@pytest.mark.gpu
def test_error_of_the_range(built_lib):
    rng = np.random.default_rng(4)
    e, v = _error(np.exp2(rng.uniform(-30, 4, 400_000)))
    assert np.all(np.abs(e) <= np.spacing(np.maximum(1.0, np.abs(v))) + 2.0 ** -58)
