"""Several charge columns in one pass (csrc/fmm.cu k_s2m_multi, k_evaluate_multi
at 8 and 16 columns a launch, and remainders of both) against the same columns
one at a time, with empty and full tiles of sources.  Both sum the same values in
other orders: bar 1e-12, the parity bar of the FP64 form."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel, params", [("Laplace_Eval", {}),
                                            ("Modified_Helmholtz_Eval", {"helmholtz_k": 3.0})])
@pytest.mark.parametrize("columns", [1, 8, 9, 16, 17, 25])
def test_columns_match_single_columns(built_lib, kernel, params, columns):
    from flexmm_b200 import KI_FMM, KI_Helper
    rng = np.random.default_rng(columns)
    n = 3000
    th = rng.uniform(0, 2 * np.pi, n)
    x, y = 0.8 * np.cos(th), 0.8 * np.sin(th)
    tx, ty = rng.uniform(-1, 1, 500), rng.uniform(-1, 1, 500)
    tau = rng.standard_normal((columns, n))
    F = KI_FMM(x, y, kernel, 70, 33, bbox=[-1.0, 1.0, -1.0, 1.0], helper=KI_Helper(), **params)
    F.build_expansions(tau)
    own, other = F.source_evaluation(x, y), F.target_evaluation(tx, ty)
    F.status()
    for k in {0, columns // 2, columns - 1}:
        F.build_expansions(tau[k])
        assert rel_l2(own[k], F.source_evaluation(x, y)) < 1e-12
        assert rel_l2(other[k], F.target_evaluation(tx, ty)) < 1e-12
