"""The level passes' launch shape (csrc/fmm.cu level_fit) depends on the number
of charge columns alone, not on which call came first in the process: one
column and several take the same shared memory a block at Nequiv <= 40 and differ
in the blocks per SM only.  The shape decides how many row blocks a tile holds
and with that the last bits, so two processes with the calls in either order
have to agree on every bit.

Points in half of the box: 512 sibling groups on the level below the root's
1024, 64 row blocks, where 148 blocks (37 a class on the way down) take two row
blocks a tile and 296 take one."""
import subprocess
import sys

import numpy as np
import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu

CHILD = """
import sys
import numpy as np
from flexmm_b200 import KI_FMM, KI_Helper
rng = np.random.default_rng(11)
n = 30_000
x, y = rng.uniform(-1, 1, n), rng.uniform(-1, 0, n)
tau = rng.standard_normal((3, n))
F = KI_FMM(x, y, "Laplace_Eval", 32, int(sys.argv[3]), bbox=[-1, 1, -1, 1], helper=KI_Helper())
out = {}
for what in sys.argv[1].split(","):
    F.build_expansions(tau[0] if what == "one" else tau)
    out[what] = F.source_evaluation(x, y)
F.status()
np.savez(sys.argv[2], **out)
"""


@pytest.mark.parametrize("neq", [16, 40])
def test_results_do_not_depend_on_the_order_of_calls(built_lib, tmp_path, neq):
    res = []
    for order in ("one,several", "several,one"):
        f = str(tmp_path / (order.replace(",", "_") + ".npz"))
        subprocess.run([sys.executable, "-c", CHILD, order, f, str(neq)], cwd=REPO, check=True,
                       timeout=300)
        res.append(np.load(f))
    for k in ("one", "several"):
        assert np.array_equal(res[0][k], res[1][k]), k
