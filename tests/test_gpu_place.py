"""A target's arithmetic is a function of its leaf alone: targets are binned into
their leaves in no particular order, and where a target lands (which target shares
its lane, which tile it is in) must not move its bits.  Here with pairs that take
the evaluation's second path (csrc/sweep.cuh): K0 and K1 from k r = 1 on, and
sources that coincide with a target."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NS = 700   # sources, all in one leaf


def _cuda(*a):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in a]


def _fmm(kernel, dipoles, **kw):
    from flexmm_b200 import KI_FMM, KI_Helper
    rng = np.random.default_rng(17)
    x, y = rng.uniform(-1, 1, NS), rng.uniform(-1, 1, NS)
    tau = rng.standard_normal((2, NS))
    xd, yd, td = _cuda(x, y, tau)
    F = KI_FMM(xd, yd, kernel, NS, 16, bbox=[-1, 1, -1, 1], helper=KI_Helper(), **kw)
    F.register_evaluator(None, None, "gradient", 3)
    if dipoles:
        F.register_upwardor("Laplace_Both_Eval", "slp+dlp")
        th = rng.uniform(0, 2 * np.pi, NS)
        F.build_expansions(td, "slp+dlp", _cuda(np.stack([np.cos(th), np.sin(th)]))[0])
    else:
        F.build_expansions(td[0].contiguous())
    return F, x, y


@pytest.mark.parametrize("n", [33, 64, 100, 128, 300])
@pytest.mark.parametrize("what", ["potential_evaluation", "gradient"])
@pytest.mark.parametrize("kernel, kw", [("Modified_Helmholtz_Eval", dict(helmholtz_k=1.3)),
                                        ("Modified_Helmholtz_Eval", dict(helmholtz_k=6.0)),
                                        ("Laplace_Eval", {}), ("dipoles", {}), ("Kernel", {})])
def test_bits_do_not_depend_on_the_place(built_lib, kernel, kw, what, n):
    dip = kernel == "dipoles"
    if what == "gradient" and kernel in ("dipoles", "Kernel"):
        pytest.skip("dipole sources and tabulated kernels evaluate potentials only")
    F, x, y = _fmm("Laplace_Eval" if dip else kernel, dip, **kw)
    rng = np.random.default_rng(n)
    tx, ty = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    on = rng.permutation(n)[: n // 3]   # a third of the targets sit on sources
    tx[on], ty[on] = x[on], y[on]
    ref = F.evaluate_to_points(*_cuda(tx, ty), what, True).cpu().numpy()
    assert np.all(np.isfinite(ref))
    for _ in range(4):
        p = rng.permutation(n)
        got = F.evaluate_to_points(*_cuda(tx[p], ty[p]), what, True).cpu().numpy()
        assert np.array_equal(got, ref[:, p])
