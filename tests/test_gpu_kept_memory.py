"""The split evaluation's scratch (8 bytes a source and the item list) is kept by
plans that evaluate at their own sources, and given back by the others at their
next build."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _used():
    import torch
    from cuda.bindings import runtime as rt
    torch.cuda.synchronize()
    err, dev = rt.cudaGetDevice()
    err, pool = rt.cudaDeviceGetDefaultMemPool(dev)
    err, v = rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
    assert err == rt.cudaError_t.cudaSuccess
    return int(v)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_scratch_of_plans_that_do_not_split(built_lib, precision):
    import torch
    from flexmm_b200 import KI_FMM, KI_Helper
    n = 400_000
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x, y, tau = (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) for _ in range(3))
    tx, ty = x[:1000].contiguous(), y[:1000].contiguous()
    F = KI_FMM(x, y, "Laplace_Eval", 64, 16, bbox=[0, 1, 0, 1], helper=KI_Helper(), precision=precision)

    def step(own):
        F.build_expansions(tau)
        F.source_evaluation(x, y) if own else F.target_evaluation(tx, ty)
        return _used()

    step(True)                      # sources, with the scratch
    with_scratch = step(True)
    step(False)                     # other points only ...
    without = step(False)           # ... the build after it gives the scratch back
    assert without <= with_scratch - 8 * n
    first = F.source_evaluation(x, y)   # still there to be asked for its sources
    assert step(True) == with_scratch
    assert torch.equal(first, F.source_evaluation(x, y))
