"""M2M and L2L of the black-box FMM by tensor factors (csrc/bbfmm.cu k_bb_shift)
against the row GEMM with the whole operator, which an operator that is no
tensor product takes: one element of M2MC is moved by 1e-13.  It multiplies one
coefficient of one child, at most the size of the others, so the potentials move
by about as much: bar 1e-12, the parity bar of the FP64 forms."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [2, 3, 7, 8, 9, 13, 16])
def test_shift_matches_whole_operator(built_lib, monkeypatch, p):
    from flexmm_b200 import bbfmm
    from flexmm_b200.bbfmm import BB_FMM, BB_Helper
    rng = np.random.default_rng(40 + p)
    n = 5000
    x = np.concatenate([rng.uniform(-1, 1, n - 1500), 0.3 + 0.01 * rng.standard_normal(1500)])
    y = np.concatenate([rng.uniform(-1, 1, n - 1500), -0.6 + 0.01 * rng.standard_normal(1500)])
    tau = rng.standard_normal(n)

    def run():
        F = BB_FMM(x, y, "Laplace_Eval", 20, p, bbox=[-1, 1, -1, 1], helper=BB_Helper())
        F.build_expansions(tau)
        return F.source_evaluation(x, y)

    factors = run()
    info = bbfmm.cheb_info

    def moved(order):
        d = info(order)
        d["M2MC"] = d["M2MC"].copy()
        d["M2MC"][-1, -1] += 1e-13
        return d

    monkeypatch.setattr(bbfmm, "cheb_info", moved)
    assert rel_l2(factors, run()) < 1e-12
