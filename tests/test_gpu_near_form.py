"""Where the mixed K0 passes use the near polynomials alone (k r <= 2,
csrc/fmm_mixed.cu): only where every distance allows it.

Bar 1e-6 relative L2 against the FP64 direct sum, the mixed form's own; the
near polynomials used from k r = 2 on are off by 3e-6 at 2.5 and 8e-5 at 3."""
import ctypes

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

K0 = "Modified_Helmholtz_Eval"


def _cuda(*a):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in a]


def _check(kernel, k, x, y, tau, ncut, rng, unbound=0):
    from flexmm_b200 import KI_FMM, KI_Helper, _lib
    from oracle.direct import direct_laplace, direct_mod_helmholtz
    F = KI_FMM(*_cuda(x, y), kernel, ncut, 32, bbox=[-1, 1, -1, 1], helper=KI_Helper(),
               precision="mixed", **({} if k is None else dict(helmholtz_k=k)))
    if unbound:
        levels = min(unbound, F._levels)
        ids = (ctypes.c_int * levels)(*([-1] * levels))
        _lib.call("fmm_plan_bind_levels", F._plan, levels, ctypes.cast(ids, ctypes.c_void_p))
    F.build_expansions(*_cuda(tau))
    direct = direct_laplace if k is None else lambda *a, **q: direct_mod_helmholtz(*a, k, **q)
    tx, ty = rng.uniform(-1, 1, 500), rng.uniform(-1, 1, 500)
    for px, py, skip in ((tx, ty, False), (x, y, True)):
        got = F.evaluate_to_points(*_cuda(px, py), "potential_evaluation", skip).cpu().numpy()[0]
        assert rel_l2(got, direct(x, y, tau, px, py, check=skip)) < 1e-6
    F.status()


@pytest.mark.parametrize("turn", [0.0, 0.3, 0.5])
def test_check_circle_at_any_angle(built_lib, monkeypatch, turn):
    """The circles' first point need not lie at angle 0 (the C API takes any)."""
    from flexmm_b200 import helpers
    whole = helpers.surfaces
    monkeypatch.setattr(helpers, "surfaces", lambda w, th: whole(w, th + 2 * np.pi * turn))
    rng = np.random.default_rng(6)
    n = 4000
    x, y, tau = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), rng.standard_normal(n)
    _check(K0, 12.0, x, y, tau, 40, rng)


@pytest.mark.parametrize("n, ncut", [(50, 64), (200, 64), (3000, 40)])
@pytest.mark.parametrize("kernel, k", [(K0, 0.3), (K0, 1.5), ("Laplace_Eval", None)])
def test_levels_without_expansions_may_be_unbound(built_lib, kernel, k, n, ncut):
    """Levels 0 and 1 carry no expansions and need no operators: a mixed plan
    with these levels unbound (fmm_plan_bind_levels, -1) evaluates leaves there."""
    rng = np.random.default_rng(n)
    x, y, tau = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), rng.standard_normal(n)
    _check(kernel, k, x, y, tau, ncut, rng, unbound=2)
