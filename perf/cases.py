"""Performance cases: what a program that uses flexmm_b200 has it do.

A case is a dict of plain values.  Its ``kind`` names the use:

* ``step``      one whole FMM from resident points: tree, expansions, potentials
                at the sources (coincident pairs skipped) and at a grid of targets;
* ``matvec``    one product of a solver iteration on a kept tree: new charges
                (and dipoles), potentials at the object's own sources;
* ``gradient``  new charges on a kept tree, potential and gradient at the sources
                and at a grid of targets;
* ``columns``   several charge columns on one tree, tree included, evaluated at
                the sources;
* ``stokes``    a batch of independent Stokes problems on kept trees: forward and
                charge adjoint;
* ``potential`` the differentiable black-box potential: forward, and the
                gradients of all five inputs;
* ``local``     near-field-only sums of a compactly supported kernel with point
                categories, on host (numpy) arrays, tree included.

Layouts (``flexmm_b200.workloads`` uses the same ones): ``uniform`` points in
[-1, 1]^2, ``clustered`` in 20 Gaussian clusters of sigma 0.01, ``circle`` on a
thin ring of radius 0.5 as boundary points lie.  ``bbox`` says whether the
program passes the box or lets the object find it.
"""
import math

import numpy as np
import torch

from flexmm_b200 import KI_FMM, KI_Helper, autograd
from flexmm_b200.batch import StokesBatch
from flexmm_b200.kernels import radial
from flexmm_b200.local_evaluator_category import LocalEvaluator


def listed():
    return [
        # the smallest whole call: a small test problem, bound by latency and launches
        dict(name="step_3k", kind="step", kernel="laplace", precision="fp64", layout="uniform",
             n=3000, grid=41, ncut=16, neq=16, bbox=True),
        # an ordinary whole call at middle accuracy
        dict(name="step_100k", kind="step", kernel="laplace", precision="fp64", layout="uniform",
             n=100_000, grid=316, ncut=64, neq=32, bbox=True),
        # the largest whole call: strongly clustered points, near full FP64 accuracy
        dict(name="step_1m", kind="step", kernel="laplace", precision="fp64", layout="clustered",
             n=1_000_000, grid=1000, ncut=64, neq=60, bbox=True),
        # the same points in the mixed form, the throughput setting
        dict(name="step_1m_mixed", kind="step", kernel="laplace", precision="mixed",
             layout="clustered", n=1_000_000, grid=1000, ncut=64, neq=24, bbox=True),
        # a screened-Poisson solve at a ragged size
        dict(name="step_k0", kind="step", kernel="k0", k=10.0, precision="fp64",
             layout="clustered", n=200_003, grid=450, ncut=64, neq=32, bbox=True),
        # the screened kernel in the mixed form
        dict(name="step_k0_mixed", kind="step", kernel="k0", k=10.0, precision="mixed",
             layout="clustered", n=1_000_000, grid=1000, ncut=64, neq=32, bbox=True),
        # a boundary-integral solver's matrix-vector product, tree kept over the iterations
        dict(name="matvec_250k", kind="matvec", kernel="laplace", layout="circle", n=250_007,
             ncut=50, neq=40, dipoles=False, bbox=False),
        # forces: potential and gradient at the particles and on a grid
        dict(name="gradient_100k", kind="gradient", kernel="laplace", layout="clustered",
             n=100_003, grid=200, ncut=32, neq=32, bbox=True),
        # many right-hand sides on one boundary
        dict(name="columns_16", kind="columns", kernel="k0", k=10.0, layout="circle", n=100_000,
             columns=16, ncut=64, neq=40, bbox=False),
        # a suspension: independent Stokes problems of very different sizes
        dict(name="stokes_batch", kind="stokes", problems=12, n_min=2000, n_max=200_000, ncut=64,
             neq=32),
        # fitting charges and positions through the black-box potential
        dict(name="potential_500k", kind="potential", kernel="laplace", n=500_000, m=250_000,
             ncut=64, p=16),
        # short-range corrections between bodies, from host arrays
        dict(name="local_100k", kind="local", n=100_003, grid=200, delta=2.0 ** -6, ncut=20,
             categories=7),
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], uniform over its logarithm, odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "matvec", "gradient", "columns", "stokes",
                       "potential", "local"])
    if kind == "step":
        kernel = rng.choice(["laplace", "laplace", "k0"])
        precision = rng.choice(["fp64", "mixed"])
        n = _between(rng, 3000, 300_000 if (kernel, precision) == ("k0", "fp64") else 1_000_000)
        case = dict(kind=kind, kernel=kernel, precision=precision,
                    layout=rng.choice(["uniform", "clustered", "circle"]), n=n,
                    grid=max(9, int(math.sqrt(n) * rng.uniform(0.3, 1.0))),
                    ncut=rng.choice([16, 32, 50, 64]),
                    neq=rng.choice([16, 24, 24, 32] if precision == "mixed" else [16, 24, 32, 40, 60]),
                    bbox=True)
        if kernel == "k0":
            case["k"] = rng.choice([1.0, 5.0, 10.0, 40.0])
        return case
    if kind == "matvec":
        kernel = rng.choice(["laplace", "laplace", "k0"])
        case = dict(kind=kind, kernel=kernel, layout=rng.choice(["uniform", "clustered", "circle"]),
                    n=_between(rng, 3000, 300_000), ncut=rng.choice([16, 32, 50, 64]),
                    neq=rng.choice([16, 24, 32, 40, 60]),
                    dipoles=kernel == "laplace" and rng.random() < 0.5, bbox=rng.random() < 0.5)
        if kernel == "k0":
            case["k"] = rng.choice([1.0, 5.0, 10.0, 40.0])
        return case
    if kind == "gradient":
        n = _between(rng, 3000, 200_000)
        case = dict(kind=kind, kernel=rng.choice(["laplace", "laplace", "k0"]),
                    layout=rng.choice(["uniform", "clustered"]), n=n,
                    grid=max(9, int(math.sqrt(n) * rng.uniform(0.3, 1.0))),
                    ncut=rng.choice([16, 32, 64]), neq=rng.choice([16, 24, 32, 40]), bbox=True)
        if case["kernel"] == "k0":
            case["k"] = rng.choice([1.0, 5.0, 10.0])
        return case
    if kind == "columns":
        kernel = rng.choice(["laplace", "k0"])
        case = dict(kind=kind, kernel=kernel, layout=rng.choice(["uniform", "circle"]),
                    n=_between(rng, 3000, 100_000), columns=rng.choice([2, 5, 8, 11, 16]),
                    ncut=rng.choice([32, 64]), neq=rng.choice([24, 32, 40]), bbox=False)
        if kernel == "k0":
            case["k"] = rng.choice([1.0, 5.0, 10.0])
        return case
    if kind == "stokes":
        n_min = _between(rng, 2000, 10_000)
        return dict(kind=kind, problems=rng.choice([1, 3, 8]), n_min=n_min,
                    n_max=_between(rng, n_min, 150_000), ncut=rng.choice([32, 64]),
                    neq=rng.choice([16, 24, 32]))
    if kind == "potential":
        n = _between(rng, 3000, 300_000)
        return dict(kind=kind, kernel="laplace", n=n, m=_between(rng, max(1000, n // 8), n),
                    ncut=rng.choice([32, 64]), p=rng.choice([8, 10, 12]))
    return dict(kind=kind, n=_between(rng, 3000, 100_000), grid=rng.randint(30, 250),
                delta=rng.choice([2.0 ** -5, 2.0 ** -6]), ncut=20, categories=rng.randint(2, 9))


# ------------------------------------------------------------------ inputs ----
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * (seed + 1))
    return g


def _uniform(g, n, lo=-1.0, hi=1.0):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _points(case, g):
    n, layout = case["n"], case["layout"]
    if layout == "uniform":
        return _uniform(g, n), _uniform(g, n)
    if layout == "clustered":
        cx, cy = _uniform(g, 20, -0.9, 0.9), _uniform(g, 20, -0.9, 0.9)
        which = torch.arange(n, device="cuda") * 20 // n
        return cx[which] + 0.01 * _normal(g, n), cy[which] + 0.01 * _normal(g, n)
    th = _uniform(g, n, 0.0, 2.0 * math.pi)
    r = 0.5 + _uniform(g, n, -1e-3, 1e-3)
    return r * torch.cos(th), r * torch.sin(th)


def _grid(case):
    half = 0.45 if case["layout"] == "circle" else 1.0
    a = torch.linspace(-half, half, case["grid"], device="cuda", dtype=torch.float64)
    gx, gy = torch.meshgrid(a, a, indexing="xy")
    return gx.reshape(-1).contiguous(), gy.reshape(-1).contiguous()


def _bbox(case):
    return [-1.0, 1.0, -1.0, 1.0] if case["bbox"] else None


_NAMES = {"laplace": "Laplace_Eval", "k0": "Modified_Helmholtz_Eval"}


def _kernel_args(case):
    return dict(helmholtz_k=case["k"]) if case["kernel"] == "k0" else {}


def _fmm(case, s):
    return KI_FMM(s["x"], s["y"], _NAMES[case["kernel"]], case["ncut"], case["neq"],
                  bbox=_bbox(case), helper=s["helper"], precision=case.get("precision", "fp64"),
                  **_kernel_args(case))


# operators that a program keeps over its calls, and the local kernel's table
_HELPERS = {}
_STOKES = {}
_BUMPS = {}


def _bump(delta):
    """(1 - r^2 / delta^2)^3 inside r < delta, tabulated as the local evaluators take it."""
    if delta not in _BUMPS:
        def f(r):
            q = 1.0 - (np.asarray(r, dtype=np.float64) / delta) ** 2
            return np.where(np.asarray(r) < delta, q * q * q, 0.0)
        _BUMPS[delta] = radial(f, 1e-30, 4.0, tol=1e-4, name="Bump")
    return _BUMPS[delta]


def _stokes_sizes(case):
    p, lo, hi = case["problems"], case["n_min"], case["n_max"]
    return [int(round(lo * (hi / lo) ** ((i + 0.5) / p))) for i in range(p)]


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "stokes":
        sizes = _stokes_sizes(case)
        points = [(_uniform(g, n), _uniform(g, n)) for n in sizes]
        # opposite corners of the box, so that every batch of this size uses the same operators
        for x, y in points:
            x[0], y[0], x[1], y[1] = -1.0, -1.0, 1.0, 1.0
        s["points"] = points
        s["forces"] = [(_normal(g, n), _normal(g, n)) for n in sizes]
        s["cotangents"] = [(_normal(g, n), _normal(g, n), _normal(g, n)) for n in sizes]
        key = case["neq"]
        s["batch"] = StokesBatch([(x.cpu().numpy(), y.cpu().numpy()) for x, y in points],
                                 Nequiv=case["neq"], Ncutoff=case["ncut"],
                                 precomputations=_STOKES.get(key))
        _STOKES[key] = s["batch"].precomputations
        return s
    if kind == "potential":
        s["inputs"] = [t.requires_grad_(True) for t in
                       (_uniform(g, case["n"]), _uniform(g, case["n"]), _normal(g, case["n"]),
                        _uniform(g, case["m"]), _uniform(g, case["m"]))]
        s["cotangent"] = _normal(g, case["m"])
        return s
    if kind == "local":
        n, c = case["n"], case["categories"]
        s["x"], s["y"] = _uniform(g, n).cpu().numpy(), _uniform(g, n).cpu().numpy()
        s["tau"] = _normal(g, n).cpu().numpy()
        s["tx"], s["ty"] = (t.cpu().numpy() for t in _grid(dict(layout="uniform", grid=case["grid"])))
        s["cat"] = torch.randint(0, c, (n,), generator=g, device="cuda").cpu().numpy()
        s["tcat"] = torch.randint(0, c, (s["tx"].size,), generator=g, device="cuda").cpu().numpy()
        s["kernel"] = _bump(case["delta"])
        return s
    s["x"], s["y"] = _points(case, g)
    if kind == "columns":
        s["tau"] = _normal(g, case["columns"], case["n"])
    elif kind == "matvec" and case["dipoles"]:
        s["tau"] = _normal(g, 2, case["n"])
        th = _uniform(g, case["n"], 0.0, 2.0 * math.pi)
        s["normals"] = torch.stack([torch.cos(th), torch.sin(th)])
    else:
        s["tau"] = _normal(g, case["n"])
    if kind in ("step", "gradient"):
        s["tx"], s["ty"] = _grid(case)
    if case["bbox"]:  # one operator set per kernel and order, as one program keeps
        key = (case["kernel"], case.get("k"), case["neq"])
        s["helper"] = _HELPERS.setdefault(key, KI_Helper())
    else:             # the box follows the points, so the operators follow the problem
        s["helper"] = KI_Helper()
    fmm = _fmm(case, s)  # forms the operators of every level this problem meets
    if kind in ("matvec", "gradient"):
        if kind == "gradient":
            fmm.register_evaluator(None, None, "gradient", 3)
        elif case["dipoles"]:
            fmm.register_upwardor("Laplace_Both_Eval", "slp+dlp")
        s["fmm"] = fmm
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        fmm = _fmm(case, s)
        fmm.build_expansions(s["tau"])
        return fmm.source_evaluation(s["x"], s["y"]), fmm.target_evaluation(s["tx"], s["ty"])
    if kind == "matvec":
        fmm = s["fmm"]
        if case["dipoles"]:
            fmm.build_expansions(s["tau"], "slp+dlp", s["normals"])
        else:
            fmm.build_expansions(s["tau"])
        return fmm.source_evaluation(s["x"], s["y"])
    if kind == "gradient":
        fmm = s["fmm"]
        fmm.build_expansions(s["tau"])
        return (fmm.evaluate_to_points(s["x"], s["y"], "gradient", True),
                fmm.evaluate_to_points(s["tx"], s["ty"], "gradient", False))
    if kind == "columns":
        fmm = _fmm(case, s)
        fmm.build_expansions(s["tau"])
        return fmm.source_evaluation(s["x"], s["y"])
    if kind == "stokes":
        # one row block per output: (u, v, p) of all problems, then (dfx, dfy) of all
        fwd = s["batch"].forward(s["forces"])
        adj = s["batch"].adjoint(s["cotangents"])
        return ([torch.cat([o[i] for o in fwd]) for i in range(3)],
                [torch.cat([o[i] for o in adj]) for i in range(2)])
    if kind == "potential":
        u = autograd.fmm_potential(*s["inputs"], kernel=_NAMES[case["kernel"]], method="bb",
                                   Ncutoff=case["ncut"], p=case["p"], bbox=[-1.0, 1.0, -1.0, 1.0])
        return u.detach(), torch.autograd.grad(u, s["inputs"], s["cotangent"])
    ev = LocalEvaluator(s["x"], s["y"], s["cat"], s["kernel"], case["delta"], ncutoff=case["ncut"])
    ev.load_tau(s["tau"])
    return (ev.target_evaluation(s["x"], s["y"], s["cat"]),
            ev.target_evaluation(s["tx"], s["ty"], s["tcat"]))


# -------------------------------------------------------------------- work ----
def work(case):
    """One pass: inputs read and outputs written once, and the kernel values
    and translations of the FMM itself (about half-full leaves, nine
    neighbouring leaves a target, 27 interactions a box)."""
    kind = case["kind"]
    value = dict(laplace=20, k0=40).get(case.get("kernel"), 30)  # operations of a kernel value
    if kind == "local":
        n, m = case["n"], case["n"] + case["grid"] ** 2
        pairs = m * n * min(1.0, math.pi * case["delta"] ** 2 / 4.0)
        return dict(bytes=8.0 * (4 * n + 4 * m), flops=10.0 * pairs)
    if kind == "stokes":
        sizes = _stokes_sizes(case)
        n, rows, value = sum(sizes), 2 * case["neq"], 60
        return dict(bytes=8.0 * 14 * n, flops=_fmm_flops(n, n, case["ncut"], case["neq"], rows, value)
                    + _fmm_flops(n, n, case["ncut"], case["neq"], rows, value)
                    + _fmm_flops(n, n, case["ncut"], case["neq"], case["neq"], 30))
    if kind == "potential":
        n, m, q = case["n"], case["m"], case["p"] ** 2
        one = _fmm_flops(n, m, case["ncut"], q / 10.0, q, value)
        back = _fmm_flops(m, n, case["ncut"], q / 10.0, q, value)
        return dict(bytes=8.0 * (3 * n + 2 * m + 2 * m + 3 * n + 2 * m), flops=2 * one + back)
    n = case["n"]
    m = case["grid"] ** 2 if kind in ("step", "gradient") else 0
    cols = case.get("columns", 1)
    outs = 3 if kind == "gradient" else 1
    extra = 3 if case.get("dipoles") else 0
    near = _fmm_flops(n, n + m, case["ncut"], case["neq"], case["neq"], value + 10 * (outs - 1) + 5 * extra)
    return dict(bytes=8.0 * (2 * n + (cols + extra) * n + 2 * m + outs * cols * (n + m)),
                flops=near + (cols - 1) * 4.0 * n * case["ncut"])


def _fmm_flops(n, m, ncut, circle, rows, value):
    boxes = 2.0 * n / ncut
    return (value * (circle * (n + m) + 4.5 * ncut * m)
            + boxes * (27 * 2 * rows ** 2 + 8 * rows ** 2))


# ------------------------------------------------------------------- exact ----
PAIRS = 2.6e11  # log pairs that a plain direct sum does in some seconds


def _sum_pairs(nt, ns, f):
    """Rows of f(i0, i1) -> tuple of [i1 - i0] (or [columns, i1 - i0]) sums, joined."""
    step = max(1, min(nt, 6_000_000 // ns))
    parts = [f(i, min(nt, i + step)) for i in range(0, nt, step)]
    return [torch.cat(p, dim=-1) for p in zip(*parts)]


def _diff(tx, ty, sx, sy, a, b):
    dx = tx[a:b, None] - sx[None, :]
    dy = ty[a:b, None] - sy[None, :]
    return dx, dy, dx * dx + dy * dy


def _potential(case, s, tx, ty, skip):
    x, y, tau = s["x"], s["y"], s["tau"]
    two = tau if tau.dim() == 2 and not case.get("dipoles") else None

    def part(a, b):
        dx, dy, d2 = _diff(tx, ty, x, y, a, b)
        same = d2 == 0 if skip else None
        if same is not None:
            d2 = d2.masked_fill(same, 1.0)
        if case["kernel"] == "laplace":
            v = torch.log(d2) * (-0.25 / math.pi)
        else:
            v = torch.special.modified_bessel_k0(case["k"] * torch.sqrt(d2)) * (0.5 / math.pi)
        if same is not None:
            v = v.masked_fill(same, 0.0)
        if two is not None:
            return (two @ v.T,)
        if case.get("dipoles"):
            w = tau[1] * s["normals"]
            return (v @ tau[0] + ((dx * w[0] + dy * w[1]) / d2).sum(1) * (0.5 / math.pi),)
        return (v @ tau,)
    return _sum_pairs(tx.numel(), x.numel(), part)[0]


def _gradient(case, s, tx, ty, skip):
    x, y, tau = s["x"], s["y"], s["tau"]

    def part(a, b):
        dx, dy, d2 = _diff(tx, ty, x, y, a, b)
        same = d2 == 0 if skip else None
        if same is not None:
            d2 = d2.masked_fill(same, 1.0)
        if case["kernel"] == "laplace":
            v = torch.log(d2) * (-0.25 / math.pi)
            w = (-0.5 / math.pi) / d2
        else:
            r = torch.sqrt(d2)
            v = torch.special.modified_bessel_k0(case["k"] * r) * (0.5 / math.pi)
            w = torch.special.modified_bessel_k1(case["k"] * r) * (-0.5 * case["k"] / math.pi) / r
        if same is not None:
            v = v.masked_fill(same, 0.0)
            w = w.masked_fill(same, 0.0)
        return v @ tau, (w * dx) @ tau, (w * dy) @ tau
    return torch.stack(_sum_pairs(tx.numel(), x.numel(), part))


def _stokes_exact(x, y, fx, fy, gp=None):
    """(u, v, p) of forces at their own points; with gp also the transposed
    pressure row, (du, dv) added by it."""
    def part(a, b):
        dx, dy, d2 = _diff(x, y, x, y, a, b)
        same = d2 == 0
        i2 = (1.0 / d2.masked_fill(same, 1.0)).masked_fill(same, 0.0)
        lg = torch.log(d2.masked_fill(same, 1.0)) * -0.5
        px, py = dx * i2, dy * i2
        xy = dx * py
        u = (lg + dx * px) @ fx + xy @ fy
        v = xy @ fx + (lg + dy * py) @ fy
        if gp is None:
            return u * (0.25 / math.pi), v * (0.25 / math.pi), (px @ fx + py @ fy) * (0.5 / math.pi)
        return (u * (0.25 / math.pi) - (px @ gp) * (0.5 / math.pi),
                v * (0.25 / math.pi) - (py @ gp) * (0.5 / math.pi))
    return _sum_pairs(x.numel(), x.numel(), part)


def exact(case, seed):
    kind = case["kind"]
    if kind == "stokes":
        if sum(float(n) ** 2 for n in _stokes_sizes(case)) > PAIRS:
            return None
        s = prepare(case, seed)
        fwd = [_stokes_exact(x, y, fx, fy) for (x, y), (fx, fy) in zip(s["points"], s["forces"])]
        adj = [_stokes_exact(x, y, gu, gv, gp)
               for (x, y), (gu, gv, gp) in zip(s["points"], s["cotangents"])]
        return ([torch.cat([o[i] for o in fwd]) for i in range(3)],
                [torch.cat([o[i] for o in adj]) for i in range(2)])
    if kind == "potential":
        if 2.0 * case["n"] * case["m"] > PAIRS:
            return None
        s = prepare(case, seed)
        sx, sy, tau, tx, ty = (t.detach() for t in s["inputs"])
        c, gu = dict(case), s["cotangent"]
        at_t = _gradient(c, dict(x=sx, y=sy, tau=tau), tx, ty, False)
        at_s = _gradient(c, dict(x=tx, y=ty, tau=gu), sx, sy, False)
        return at_t[0], (tau * at_s[1], tau * at_s[2], at_s[0], gu * at_t[1], gu * at_t[2])
    if kind == "local":
        if float(case["n"]) * (case["n"] + case["grid"] ** 2) > PAIRS:
            return None
        s = prepare(case, seed)
        d = {k: torch.from_numpy(s[k]).cuda() for k in ("x", "y", "tau", "tx", "ty", "cat", "tcat")}

        def near(tx, ty, tcat):
            def part(a, b):
                d2 = _diff(tx, ty, d["x"], d["y"], a, b)[2]
                q = (1.0 - d2 / case["delta"] ** 2).clamp_min(0.0)
                return ((q * q * q).masked_fill(tcat[a:b, None] == d["cat"][None, :], 0.0) @ d["tau"],)
            return _sum_pairs(tx.numel(), d["x"].numel(), part)[0]
        return (near(d["x"], d["y"], d["cat"]).cpu().numpy(),
                near(d["tx"], d["ty"], d["tcat"]).cpu().numpy())
    n, m = case["n"], case["grid"] ** 2 if kind in ("step", "gradient") else 0
    if float(n) * (n + m) * (3.0 if case["kernel"] == "k0" else 1.0) > PAIRS:
        return None
    s = prepare(case, seed)
    if kind == "step":
        return (_potential(case, s, s["x"], s["y"], True),
                _potential(case, s, s["tx"], s["ty"], False))
    if kind == "gradient":
        return (_gradient(case, s, s["x"], s["y"], True),
                _gradient(case, s, s["tx"], s["ty"], False))
    return _potential(case, s, s["x"], s["y"], True)
