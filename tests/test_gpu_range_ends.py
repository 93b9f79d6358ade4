"""Gradients at the ends of the double range, where a squared distance or a
squared screening constant leaves it but the gradient does not: one unit charge
at the origin, a target on the x axis.  Bar 4e-15 relative: a few roundings."""
import numpy as np
import pytest
from scipy.special import k1e

pytestmark = pytest.mark.gpu


def _gradient(kernel, x, method="ki", **kw):
    import torch
    from flexmm_b200 import BB_FMM, BB_Helper, KI_FMM, KI_Helper
    o = torch.zeros(1, dtype=torch.float64).cuda()
    box = dict(bbox=[-1, 1, -1, 1], **kw)
    F = (KI_FMM(o, o.clone(), kernel, 8, 16, helper=KI_Helper(), **box) if method == "ki" else
         BB_FMM(o, o.clone(), kernel, 8, 6, helper=BB_Helper(), **box))
    F.register_evaluator(None, None, "gradient", 3)
    F.build_expansions(torch.ones(1, dtype=torch.float64).cuda())
    xd = torch.from_numpy(x).cuda()
    g = F.evaluate_to_points(xd, torch.zeros_like(xd), "gradient", False).cpu().numpy()
    assert np.all(g[2] == 0)
    return g[1] * (2 * np.pi)


def test_laplace_gradient_at_large_distances(built_lib):
    """d^2 up to 2^1022: its reciprocal is still a normal number."""
    top = 2.0 ** 511
    x = np.concatenate([top * (1 - 2.0 ** -np.arange(2, 53)), top * np.linspace(0.7, 0.999, 200),
                        [2.0 ** 510, 2.0 ** 510 * (1 - 2.0 ** -52), 1e150]])
    got = _gradient("Laplace_Eval", x)
    assert np.max(np.abs(got * -x - 1)) < 4e-15


@pytest.mark.parametrize("method", ["ki", "bb"])
@pytest.mark.parametrize("k", [1e-200, 1e-170, 1e-160, 1e-156, 1e-150, 1e-100, 1e-8])
def test_k0_gradient_of_small_constants(built_lib, k, method):
    """K0(k r)' = -k K1(k r): -1 / r where k r is small, whatever k^2 is."""
    x = np.array([1e-3, 0.3, 1.0, 50.0])
    got = _gradient("Modified_Helmholtz_Eval", x, method, helmholtz_k=k)
    want = -k * k1e(k * x) * np.exp(-k * x)
    assert np.max(np.abs(got / want - 1)) < 4e-15
