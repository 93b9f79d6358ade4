"""The evaluation items of the FP64 forms (csrc/items.cuh) at the sizes where
their split changes: one leaf (Ncutoff >= N, so the evaluation is the direct
sum) holding n points, n around the 32-target tiles, the 128-target items and
the 512-source chunks, against the C oracle's FP64 direct sum.

Bar: each of the n terms of a sum carries a few roundings (distance, kernel
value, product) and the sum n more, so the error of a target is at most
(n + 16) ulp of the sum of its terms' absolute values."""
import numpy as np
import pytest

from oracle.direct import direct_laplace, direct_laplace_grad, direct_mod_helmholtz, \
    direct_mod_helmholtz_grad

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 5, 16, 31, 32, 33, 63, 64, 65, 97, 127, 128, 129, 161, 511, 512, 513, 700]
EPS = np.finfo(np.float64).eps


def _points(n, seed):
    rng = np.random.default_rng(seed)
    x, y, tau = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), rng.standard_normal(n)
    if n > 4:  # two coincident pairs
        x[1], y[1], x[n - 1], y[n - 1] = x[0], y[0], x[2], y[2]
    return x, y, tau


def _fmm(x, y, kernel, n, **kw):
    import torch
    from flexmm_b200 import KI_FMM, KI_Helper
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    return KI_FMM(xd, yd, kernel, max(n, 1), 16, bbox=[-1, 1, -1, 1], helper=KI_Helper(), **kw), xd, yd


def _within(got, want, scale, n):
    err = np.abs(np.asarray(got) - want)
    assert np.all(err <= (n + 16) * EPS * scale + 1e-300), (err / scale).max() / EPS


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kernel", ["Laplace_Eval", "Modified_Helmholtz_Eval"])
def test_one_leaf_is_the_direct_sum(built_lib, n, kernel):
    import torch
    x, y, tau = _points(n, n)
    kw = {} if kernel == "Laplace_Eval" else dict(helmholtz_k=3.0)
    F, xd, yd = _fmm(x, y, kernel, n, **kw)
    F.register_evaluator(None, None, "gradient", 3)
    F.build_expansions(torch.from_numpy(tau).cuda())
    rng = np.random.default_rng(1000 + n)
    tx, ty = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    txd, tyd = torch.from_numpy(tx).cuda(), torch.from_numpy(ty).cuda()
    if kernel == "Laplace_Eval":
        pot, grad = direct_laplace, direct_laplace_grad
    else:
        pot = lambda *a, **k: direct_mod_helmholtz(*a, 3.0, **k)
        grad = lambda *a, **k: direct_mod_helmholtz_grad(*a, 3.0, **k)
    a = np.abs(tau)
    for px, py, got, skip in ((x, y, F.source_evaluation(xd, yd), True),
                              (tx, ty, F.target_evaluation(txd, tyd), False)):
        # |log| changes sign at distance 1: bound the terms by |K| + 1
        scale = np.abs(pot(x, y, a, px, py, check=skip)) + a.sum()
        _within(got.cpu().numpy(), pot(x, y, tau, px, py, check=skip), scale, n)
    for px, py, q, skip in ((x, y, (xd, yd), True), (tx, ty, (txd, tyd), False)):
        got = F.evaluate_to_points(*q, "gradient", skip).cpu().numpy()
        want = np.asarray(grad(x, y, tau, px, py, check=skip))
        dx, dy = px[:, None] - x, py[:, None] - y
        r = np.hypot(dx, dy)
        # |grad K| <= c / r for both kernels (c = 1/(2 pi), x K1(x) <= 1); the
        # difference of two coordinates of size 1 carries their rounding / r
        w = np.where(r > 0, 1 / np.where(r > 0, r, 1), 0.0)
        scale = (w * (1 + w * EPS) * a).sum(1) + a.sum()
        for k in range(3):
            _within(got[k], want[k], scale, n)


@pytest.mark.parametrize("n", [33, 64, 100, 128, 300])
def test_binned_targets_do_not_depend_on_their_place(built_lib, n):
    """The targets of a leaf stand in no particular order: the same target
    gives the same bits wherever it lands in the leaf's items."""
    import torch
    x, y, tau = _points(700, 3)
    F, _, _ = _fmm(x, y, "Laplace_Eval", 700)
    F.build_expansions(torch.from_numpy(tau).cuda())
    rng = np.random.default_rng(n)
    tx, ty = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    ref = F.target_evaluation(torch.from_numpy(tx).cuda(), torch.from_numpy(ty).cuda()).cpu().numpy()
    for _ in range(3):
        p = rng.permutation(n)
        got = F.target_evaluation(torch.from_numpy(tx[p]).cuda(), torch.from_numpy(ty[p]).cuda())
        assert np.array_equal(got.cpu().numpy(), ref[p])


@pytest.mark.parametrize("n", SIZES)
def test_one_leaf_black_box(built_lib, n):
    import torch
    from flexmm_b200.bbfmm import BB_FMM, BB_Helper
    x, y, tau = _points(n, n + 50)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    F = BB_FMM(xd, yd, "Laplace_Eval", n, 4, bbox=[-1, 1, -1, 1], helper=BB_Helper())
    F.register_evaluator(None, None, "gradient", 3)
    F.build_expansions(torch.from_numpy(tau).cuda())
    scale = np.abs(direct_laplace(x, y, np.abs(tau), x, y, check=True)) + np.abs(tau).sum()
    _within(F.source_evaluation(xd, yd).cpu().numpy(), direct_laplace(x, y, tau, x, y, check=True),
            scale, n)
    want = np.asarray(direct_laplace_grad(x, y, tau, x, y, check=True))
    r = np.hypot(x[:, None] - x, y[:, None] - y)
    w = np.where(r > 0, 1 / np.where(r > 0, r, 1), 0.0)
    got = F.evaluate_to_points(xd, yd, "gradient", True).cpu().numpy()
    for k in range(3):
        _within(got[k], want[k], (w * (1 + w * EPS) * np.abs(tau)).sum(1) + np.abs(tau).sum(), n)


@pytest.mark.parametrize("dipoles", [False, True])
@pytest.mark.parametrize("n", SIZES + [383, 384, 385])
def test_one_leaf_stokes(built_lib, n, dipoles):
    import torch
    from flexmm_b200.stokes import FMM
    from oracle.direct import direct_stokes, direct_stokes_dipole
    x, y, fx = _points(n, n + 90)
    rng = np.random.default_rng(n)
    fy, gx, gy = (rng.standard_normal(n) for _ in range(3))
    th = rng.uniform(0, 2 * np.pi, n)
    nx, ny = np.cos(th), np.sin(th)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    F = FMM(xd, yd, 8, max(n, 1), [-1, 1, -1, 1])
    c = lambda *a: [torch.from_numpy(v).cuda() for v in a]
    if dipoles:
        F.build_expansions_dipole(*c(fx, fy, gx, gy, nx, ny))
        want = direct_stokes_dipole(x, y, fx, fy, gx, gy, nx, ny, x, y, True)
    else:
        F.build_expansions(*c(fx, fy))
        want = direct_stokes(x, y, fx, fy, x, y, True)
    got = [v.cpu().numpy() for v in F.evaluate_to_points(xd, yd, True)]
    # a pair's terms are at most (|log r| + 1 + 1/r) |f| and, for stresslets,
    # (4/r + 4/r^2) |sigma|, over 4 pi (u, v) and 2 pi (p): all within
    # (2 + 1/r)|f| + (4/r + 4/r^2)|sigma|; the difference of two coordinates
    # carries their rounding / r, up to four times over
    r = np.hypot(x[:, None] - x, y[:, None] - y)
    w = np.where(r > 0, 1 / np.where(r > 0, r, 1), 0.0)
    s = (2 + w) * (1 + 4 * w * EPS) * (np.abs(fx) + np.abs(fy))
    if dipoles:
        s = s + (4 * w + 4 * w * w) * (1 + 4 * w * EPS) * (np.abs(gx) + np.abs(gy))
    for k in range(3):
        _within(got[k], want[k], s.sum(1), n)
