"""FP64 S2M and its solve (csrc/fmm.cu k_s2m, k_s2m_multi, k_c2e_leaves) where
the check points split differently over the lanes (up to 32, up to 48, more),
leaves of more than one staged chunk, one column and a second column group,
against the oracle's KIFMM.  Bar 1e-12, the parity bar of the FP64 form."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle.kernels import laplace
from oracle.kifmm import KIFMM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("neq", [5, 32, 33, 48, 49, 63])
def test_s2m_matches_oracle(built_lib, neq):
    from flexmm_b200 import KI_FMM, KI_Helper
    rng = np.random.default_rng(100 + neq)
    n = 6000 + neq
    x = np.concatenate([rng.uniform(-1, 1, n - 1500), -0.4 + 0.01 * rng.standard_normal(1500)])
    y = np.concatenate([rng.uniform(-1, 1, n - 1500), 0.3 + 0.01 * rng.standard_normal(1500)])
    tau = rng.standard_normal((9, n))
    bbox = [-1.0, 1.0, -1.0, 1.0]
    F = KI_FMM(x, y, "Laplace_Eval", 150, neq, bbox=bbox, helper=KI_Helper())
    O = KIFMM(x, y, laplace, 150, neq, bbox=bbox)
    O.build_expansions(tau[8])
    want = O.source_evaluation(x, y)
    F.build_expansions(tau[8])
    assert rel_l2(F.source_evaluation(x, y), want) < 1e-12
    F.build_expansions(tau)
    got = F.source_evaluation(x, y)
    F.status()
    assert rel_l2(got[8], want) < 1e-12
