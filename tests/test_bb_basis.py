"""The common basis of the black-box M2L operators (flexmm_b200/bbfmm.py
_find_basis): what it reproduces, and the device path through it against the
path through the operators themselves."""
import numpy as np
import pytest

from conftest import rel_l2
from flexmm_b200 import _lib
from flexmm_b200.bbfmm import BBPrecomputation, cheb_info
from flexmm_b200.kernels import Laplace, ModifiedHelmholtz


@pytest.mark.parametrize("p, kernel, width", [(9, Laplace(), 0.5), (10, Laplace(), 2.0 ** -9),
                                              (12, ModifiedHelmholtz(5.0), 0.25),
                                              (16, Laplace(), 2.0 ** -4)])
def test_basis_reproduces_the_operators(p, kernel, width):
    """M2L_o - Q core_o Q^T: the basis drops singular values below 1e-16 of the
    largest, so an entry moves by a few 1e-16 of the largest operator's norm."""
    pre = BBPrecomputation(width, p, kernel, cheb_info(p))
    assert pre.q is not None and pre.q.shape[1] <= _lib.BB_MAX_RANK < p * p
    assert np.abs(pre.q.T.dot(pre.q) - np.eye(pre.q.shape[1])).max() < 1e-14
    big = max(np.linalg.norm(a.dot(b), 2) for a, b in zip(pre.m2l_a, pre.m2l_b) if a is not None)
    for a, b, c in zip(pre.m2l_a, pre.m2l_b, pre.core):
        assert (a is None) == (c is None)
        if a is not None:
            assert np.linalg.norm(a.dot(b) - pre.q.dot(c).dot(pre.q.T), 2) < 2e-15 * big


def test_small_orders_need_no_basis():
    pre = BBPrecomputation(0.5, 8, Laplace(), cheb_info(8))
    assert pre.q is None and pre.core is None


@pytest.mark.gpu
@pytest.mark.parametrize("p", [7, 8, 9, 12, 16])
def test_basis_path_matches_operator_path(built_lib, monkeypatch, p):
    """The same points through the basis (p > 8) or the fragments (p <= 8) and
    through the stacked operators (a set with one width lacking a basis): bar
    1e-12, the parity bar of the FP64 forms."""
    from flexmm_b200.bbfmm import BB_FMM, BB_Helper
    rng = np.random.default_rng(p)
    n = 6000
    x, y, tau = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), rng.standard_normal(n)
    tx, ty = rng.uniform(-1, 1, 700), rng.uniform(-1, 1, 700)

    def run():
        F = BB_FMM(x, y, "Laplace_Eval", 24, p, bbox=[-1, 1, -1, 1], helper=BB_Helper())
        F.build_expansions(tau)
        return F.source_evaluation(x, y), F.target_evaluation(tx, ty)

    fast = run()
    if p > 8:
        monkeypatch.setattr(BBPrecomputation, "_find_basis", lambda self, n: None)
    slow = run()
    for a, b in zip(fast, slow):
        assert rel_l2(a, b) < 1e-12
