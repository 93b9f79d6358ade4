"""The tree build's scans (csrc/scan.cuh, tree.cu SplitScan, ParentScan, UpScan)
at the edges of their tiles: one block, the first size of several blocks, the
small tiles' last size and the first of the large ones, several tiles a block;
and the root alone.  Whole numbers: equal to the oracle's tree."""
import numpy as np
import pytest

import canon

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ncut", [(1, 1), (24, 24), (25, 24), (4096, 1), (4097, 2), (40000, 3),
                                    (151552, 40), (151553, 40)])
def test_tree_at_scan_tile_edges(built_lib, n, ncut):
    from flexmm_b200 import KI_FMM, KI_Helper
    from oracle.tree import Tree
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    k = n // 3
    x[:k], y[:k] = 0.2 + 0.01 * rng.standard_normal(k), -0.5 + 0.01 * rng.standard_normal(k)
    F = KI_FMM(x, y, "Laplace_Eval", ncut, 8, bbox=[-1.0, 1.0, -1.0, 1.0], helper=KI_Helper())
    ot = Tree(x, y, ncut, F.bbox)
    a = canon.canonical(F.tree, triples_fn=canon.gpu_triples, nonempty_sources=True)
    b = canon.canonical(ot, nonempty_sources=True)
    assert canon.compare(a, b) == []
