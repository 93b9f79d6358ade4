"""What a level pass leaves whose bounded wait ran out (grid barrier, operator
copy): the plan's flag, here set from the host.  Every evaluation of those
expansions gives NaN, status() raises, and the next build starts afresh."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(n=5000):
    import torch
    from flexmm_b200 import KI_FMM, KI_Helper
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    x, y = (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 2 - 1 for _ in range(2))
    tau = torch.randn(2, n, generator=g, device="cuda", dtype=torch.float64)
    F = KI_FMM(x, y, "Laplace_Eval", 32, 16, bbox=[-1, 1, -1, 1], helper=KI_Helper())
    F.register_evaluator(None, None, "gradient", 3)
    F.register_upwardor("Laplace_Both_Eval", "slp+dlp")
    return F, x, y, tau


def _fail(F):
    import torch
    from flexmm_b200 import _lib
    _lib.call("fmm_diag_fail_passes", F._plan,
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))


def _noalloc(F, x, y):
    import torch
    from flexmm_b200 import _lib
    out = torch.zeros_like(x)
    _lib.call("fmm_evaluate_noalloc", F._plan, ctypes.c_void_p(x.data_ptr()),
              ctypes.c_void_p(y.data_ptr()), x.numel(), 1, ctypes.c_void_p(out.data_ptr()),
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return out


BUILD = {
    "charges": lambda F, tau: F.build_expansions(tau[0].contiguous()),
    "dipoles": lambda F, tau: F.build_expansions(tau, "slp+dlp", tau),
    "columns": lambda F, tau: F.build_expansions(tau),
}
EVALUATE = {
    "sources": lambda F, x, y: F.source_evaluation(x, y),
    "targets": lambda F, x, y: F.target_evaluation(x[:777].contiguous(), y[:777].contiguous() * 0.9),
    "gradient": lambda F, x, y: F.evaluate_to_points(x, y, "gradient", True),
    "noalloc": _noalloc,
}


@pytest.mark.parametrize("build, evaluate", [("charges", e) for e in EVALUATE] +
                         [("dipoles", "sources"), ("dipoles", "targets"),
                          ("columns", "sources"), ("columns", "targets")])
def test_failed_passes_show(built_lib, build, evaluate):
    import torch
    F, x, y, tau = _case()
    BUILD[build](F, tau)
    want = EVALUATE[evaluate](F, x, y)
    F.status()
    assert torch.isfinite(want).all()
    _fail(F)
    assert torch.isnan(EVALUATE[evaluate](F, x, y)).all()
    with pytest.raises(Exception, match="level pass"):
        F.status()
    BUILD[build](F, tau)
    got = EVALUATE[evaluate](F, x, y)
    F.status()
    assert torch.equal(got, want)


def test_only_built_fp64_expansions_can_be_marked(built_lib):
    from flexmm_b200 import KI_FMM, KI_Helper, _lib
    F, x, y, tau = _case(300)
    with pytest.raises(Exception):
        _fail(F)
    M = KI_FMM(x, y, "Laplace_Eval", 32, 16, bbox=[-1, 1, -1, 1], helper=KI_Helper(), precision="mixed")
    M.build_expansions(tau[0].contiguous())
    with pytest.raises(Exception):
        _fail(M)
    M.status()
