"""K0 and K1 of the modified Helmholtz passes (csrc/bessel.cuh) where their
forms change: the series' end x = 1, the table's octaves and their eighths,
the table's end x = 1024, and distances whose squares leave the double range.

One unit charge at the origin, k = 1, targets on the x axis: the potential is
K0(x) / (2 pi), its x derivative -K1(x) / (2 pi).  Bar 4e-15 relative: a few
roundings here (exponential, polynomial, product) and scipy's own peak error
(1.2e-15 for k0, k1 in Cephes)."""
import numpy as np
import pytest
from scipy.special import k0e, k1e

pytestmark = pytest.mark.gpu


def _eval(x, k):
    import torch
    from flexmm_b200 import KI_FMM, KI_Helper, direct_evaluation
    o = torch.zeros(1, dtype=torch.float64).cuda()
    q = torch.ones(1, dtype=torch.float64).cuda()
    F = KI_FMM(o, o.clone(), "Modified_Helmholtz_Eval", 8, 16, bbox=[-1, 1, -1, 1], helper=KI_Helper(),
               helmholtz_k=k)
    F.register_evaluator(None, None, "gradient", 3)
    F.build_expansions(q)
    xd = torch.from_numpy(x).cuda()
    z = torch.zeros_like(xd)
    s = 2 * np.pi
    return (F.target_evaluation(xd, z).cpu().numpy() * s,
            F.evaluate_to_points(xd, z, "gradient", False).cpu().numpy() * s,
            direct_evaluation("Modified_Helmholtz_Eval", o, o, q, xd, z, helmholtz_k=k).cpu().numpy() * s)


def test_k0_k1_at_the_forms_edges(built_lib):
    edges = np.concatenate([2.0 ** j * (1 + np.arange(8) / 8) for j in range(10)])
    x = np.concatenate([np.nextafter(edges, 0), edges, np.nextafter(edges, 2000), edges * 1.03,
                        np.logspace(-12, 0, 200, endpoint=False), [1023.0]])
    x = x[x < 700]  # beyond, the values leave the normal range
    u, g, d = _eval(x, 1.0)
    k0, k1 = k0e(x) * np.exp(-x), k1e(x) * np.exp(-x)
    for got, want in ((u, k0), (g[0], k0), (d, k0), (-g[1], k1)):
        assert np.max(np.abs(got / want - 1)) < 4e-15
    assert np.all(g[2] == 0)


def test_k0_outside_the_table_and_the_squares_range(built_lib):
    x = np.array([1024.0, np.nextafter(1024.0, 0), 5000.0, 1e200])
    u, g, d = _eval(x, 1.0)
    assert np.all(np.abs(u) <= 1e-300) and np.all(np.abs(d) <= 1e-300) and np.all(np.isfinite(g))
    # k r is an ordinary number, (k r)^2's factors are not
    u, _, d = _eval(np.array([2e-170, 0.5e-170]), 1e170)
    want = k0e([2.0, 0.5]) * np.exp([-2.0, -0.5])
    # the squared distance underflows to 0, as it always did: K0(0) = inf
    assert np.all(np.isposinf(u) | (np.abs(u / want - 1) < 4e-15))
    u, _, d = _eval(np.array([2e150, 0.5e150]), 1e-150)
    assert np.max(np.abs(u / want - 1)) < 4e-15 and np.max(np.abs(d / want - 1)) < 4e-15
