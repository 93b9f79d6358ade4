"""The split evaluation's scratch, kept by the plan: evaluations of one plan in a
row on two streams without a wait between them, across rebuilt expansions and
after dropping them, equal the evaluation of a fresh plan bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [700, 30000])
def test_kept_scratch_equals_fresh_plan(built_lib, precision, n):
    import torch
    from flexmm_b200 import KI_FMM, KI_Helper
    rng = np.random.default_rng(n)
    x, y = (torch.from_numpy(rng.uniform(-1, 1, n)).cuda() for _ in range(2))
    taus = [torch.from_numpy(rng.standard_normal(n)).cuda() for _ in range(3)]
    helper = KI_Helper()

    def plan():
        return KI_FMM(x, y, "Laplace_Eval", 30, 24, bbox=[-1.0, 1.0, -1.0, 1.0], helper=helper,
                      precision=precision)

    want = []
    for t in taus:
        F = plan()
        F.build_expansions(t)
        want.append(F.source_evaluation(x, y).clone())
        torch.cuda.synchronize()
    F = plan()
    other = torch.cuda.Stream()
    got = []
    for k in (0, 1, 2, 1, 0):
        F.build_expansions(taus[k])
        a = F.source_evaluation(x, y)
        other.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(other):
            b = F.source_evaluation(x, y)
        torch.cuda.current_stream().wait_stream(other)
        got.append((k, a, b))
        if k == 2:
            F.drop_expansions()
    torch.cuda.synchronize()
    F.status()
    for k, a, b in got:
        assert torch.equal(a, want[k]) and torch.equal(b, want[k])
