"""The Stokes passes at every operator size their kernels split differently
(np = 24 .. 136: a warp a column block, the KIFMM's M2L up to 72, row GEMMs above)
against the same passes written out in numpy with the same host operators and the
tree's lists.  Bar 1e-12, the parity bar of the FP64 forms."""
import numpy as np
import pytest

from conftest import rel_l2
from flexmm_b200.helpers import width_key

PARITY = 1e-12


def _solve(svd, b):
    return ((b @ svd.U) * svd.SI) @ svd.VH


def _numpy_fmm(F, tree, x, y, fx, fy):
    """(u, v, p) at the sources (stokes_fmm.py:550-858), u and v unscaled alike."""
    from flexmm_b200.helpers import offsets
    from flexmm_b200.stokes import stokes_form
    from oracle.direct import direct_stokes
    n2, n1 = 2 * F.Nequiv, 2 * F.Nequiv + 1
    x, y, fx, fy = (a[tree.ordv] for a in (x, y, fx, fy))
    pre = [F.precomputations[width_key(w)] for w in F._widths]
    mult = [np.zeros((lv.n_node, n1)) for lv in tree.Levels]
    for m in range(tree.levels - 1, 1, -1):
        lv, op = tree.Levels[m], pre[m]
        for g in np.flatnonzero(lv.compute_upwards):
            s = slice(lv.bot_ind[g], lv.top_ind[g])
            form = stokes_form(x[s] - lv.xmid[g], y[s] - lv.ymid[g], op.large_x, op.large_y)
            check = form @ np.concatenate([fx[s], fy[s]])
            check[-1] = 0.0
            mult[m][g] = _solve(op.e2c, check)
        if m + 1 < tree.levels:
            kids = mult[m + 1][:, :n2].reshape(-1, 4 * n2)
            mult[m][tree.Levels[m + 1].parent_ind[::4]] = _solve(op.e2c, kids @ op.m2mc.T)
    grid = {(a + 3) * 7 + b + 3: o for o, (a, b) in enumerate(offsets())}
    loc = [np.zeros((lv.n_node, n1)) for lv in tree.Levels]
    for m in range(2, tree.levels):
        lv, op = tree.Levels[m], pre[m]
        ple = np.zeros((lv.n_node, n1))
        t, o, s = tree.interaction_triples(m).T
        for k in np.unique(o):
            i = o == k
            a, b = op.m2l_a[grid[k]], op.m2l_b[grid[k]]
            if a is not None:
                ple[t[i]] += mult[m][s[i]][:, :n2] @ (a if b is None else a @ b).T
        real = ~lv.fake_leaf
        if m > 2:
            up = loc[m - 1][lv.parent_ind[::4], :n2] @ pre[m - 1].l2lc.T
            ple += up.reshape(-1, n1)
        loc[m][real] = _solve(op.c2e, ple[real])
        loc[m][:, n2:] = 0.0
    out = np.zeros((3, x.size))
    for m, lv in enumerate(tree.Levels):
        for g in np.flatnonzero(lv.leaf & (lv.ns > 0)):
            t = slice(lv.bot_ind[g], lv.top_ind[g])
            near = [np.arange(lv.bot_ind[c], lv.top_ind[c]) for c in lv.colleagues[g] if c >= 0]
            j = np.concatenate(near)
            out[:, t] += direct_stokes(x[j], y[j], fx[j], fy[j], x[t], y[t], True)
            if m >= 2:
                f = loc[m][g]
                out[:, t] += direct_stokes(pre[m].large_x + lv.xmid[g], pre[m].large_y + lv.ymid[g],
                                           f[:F.Nequiv].copy(), f[F.Nequiv:n2].copy(), x[t], y[t], False)
    res = np.empty_like(out)
    res[:, tree.ordv] = out
    return res


@pytest.mark.gpu
@pytest.mark.parametrize("neq", [8, 12, 16, 20, 24, 28, 32, 35, 36, 43, 48, 56, 64])
def test_passes_match_numpy(built_lib, neq):
    from flexmm_b200 import KI_FMM, KI_Helper
    from flexmm_b200.stokes import FMM
    rng = np.random.default_rng(neq)
    n = 2500
    x = np.concatenate([rng.uniform(-1, 1, n - 500), 0.4 + 0.01 * rng.standard_normal(500)])
    y = np.concatenate([rng.uniform(-1, 1, n - 500), -0.7 + 0.01 * rng.standard_normal(500)])
    fx, fy = rng.standard_normal(n), rng.standard_normal(n)
    box = [-1.0, 1.0, -1.0, 1.0]
    F = FMM(x, y, neq, 20, box)
    F.build_expansions(fx, fy)
    got = F.evaluate_to_points(x, y, True)
    F.status()
    tree = KI_FMM(x, y, "Laplace_Eval", 20, 8, bbox=box, helper=KI_Helper()).tree
    assert tree.bbox == list(F.bbox)
    want = _numpy_fmm(F, tree, x, y, fx, fy)
    for a, b in zip(got, want):
        assert rel_l2(a, b) < PARITY
