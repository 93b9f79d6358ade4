"""An M2M operator that is off a tensor product by more than the Chebyshev shift's
own rounding (5e-15 of its largest element at most, p = 2 .. 16) is applied as it
is given: its result is the row GEMM's (as for any other operator), not the
factors', which do not know of the element that was moved."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("p", [4, 9, 16])
def test_moved_operator_is_applied_as_given(built_lib, monkeypatch, p):
    from flexmm_b200 import bbfmm
    from flexmm_b200.bbfmm import BB_FMM, BB_Helper
    rng = np.random.default_rng(60 + p)
    n = 4000
    x, y, tau = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), rng.standard_normal(n)
    info = bbfmm.cheb_info

    def run(by):
        def moved(order):
            d = info(order)
            d["M2MC"] = d["M2MC"].copy()
            d["M2MC"][-1, -1] += by * np.abs(d["M2MC"]).max()
            return d

        monkeypatch.setattr(bbfmm, "cheb_info", moved)
        F = BB_FMM(x, y, "Laplace_Eval", 16, p, bbox=[-1, 1, -1, 1], helper=BB_Helper())
        F.build_expansions(tau)
        return F.source_evaluation(x, y)

    factors, whole = run(0.0), run(1e-10)
    near = run(1.2e-14)
    # the two routes round differently, so which one ran shows in the bits
    assert not np.array_equal(factors, near)
    assert np.abs(near - whole).max() <= np.abs(whole).max() * 1e-8


def test_the_shift_itself_is_a_product():
    """What cheb_info forms is a product to the bar."""
    from flexmm_b200.bbfmm import cheb_info
    for p in range(2, 17):
        m, n = cheb_info(p)["M2MC"], p * p
        big = np.abs(m).max()
        for c in range(4):
            b = m[:, c * n:(c + 1) * n].reshape(p, p, p, p)
            prod = np.einsum("ac,bd->abcd", b[:, 0, :, 0], b[0, :, 0, :])
            assert np.abs(b - prod).max() <= 6e-15 * big
