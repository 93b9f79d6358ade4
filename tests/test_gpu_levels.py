"""The FP64 level passes (csrc/fmm.cu k_up_levels, k_down_levels) at every
operator size their tiles split differently (np = 8 .. 64: k parts, one or two
row blocks, one or two blocks per SM), single and several charge columns,
against the oracle's KIFMM.  Bar 1e-12, the parity bar of the FP64 form."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle.kernels import laplace
from oracle.kifmm import KIFMM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("neq", [6, 8, 13, 16, 24, 31, 40, 48, 56, 64])
def test_level_passes_match_oracle(built_lib, neq):
    from flexmm_b200 import KI_FMM, KI_Helper
    rng = np.random.default_rng(neq)
    n = 2300 + neq
    x = np.concatenate([rng.uniform(-1, 1, n - 600), 0.3 + 0.004 * rng.standard_normal(600)])
    y = np.concatenate([rng.uniform(-1, 1, n - 600), -0.2 + 0.004 * rng.standard_normal(600)])
    tau = rng.standard_normal((6, n))  # six columns: the larger M2L tiles
    bbox = [-1.0, 1.0, -1.0, 1.0]
    F = KI_FMM(x, y, "Laplace_Eval", 12, neq, bbox=bbox, helper=KI_Helper())
    O = KIFMM(x, y, laplace, 12, neq, bbox=bbox)
    want = []
    for t in tau:
        O.build_expansions(t)
        want.append(O.source_evaluation(x, y))
    F.build_expansions(tau[0])
    assert rel_l2(F.source_evaluation(x, y), want[0]) < 1e-12
    F.build_expansions(tau)
    got = F.source_evaluation(x, y)
    F.status()
    for k in range(6):
        assert rel_l2(got[k], want[k]) < 1e-12
