"""The coarsest level is solved on its interior nodes: hierarchies of one level
with no, one and many interior nodes, and values on the boundary, against a
dense solve of the assembled operator (solved to 1e-12; its condition is below
1e4: 1e-8 of the largest value)."""
import numpy as np
import pytest

from dendro_gb300 import MultiGrid, Octree

from .test_gpu_families import DEPTH, _tree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("level,split", [(0, 0), (1, 0), (1, 3), (2, 0), (2, 40), (3, 100)])
def test_one_level(ctx, oracle, level, split, precision):
    octs = _tree(level, split, seed=split)
    mg = MultiGrid(Octree.from_numpy(octs, DEPTH, ctx=ctx), max_coarse_elems=len(octs))
    assert len(mg.sizes) == 1
    oda = oracle.DA(octs, DEPTH)
    xyz = np.asarray(mg.level_nodes(0))
    og, oo = np.lexsort(xyz.T[::-1]), np.lexsort(oda.node_xyz.T[::-1])
    assert np.array_equal(xyz[og], oda.node_xyz[oo])
    n = len(xyz)
    eye = np.eye(n)
    a = np.empty((n, n))  # in the oracle's numbering, column by column
    for j in range(n):
        a[:, j] = oda.dirichlet_matvec(eye[j])
    b = np.random.Generator(np.random.PCG64(7)).uniform(-1, 1, n)
    want = np.linalg.solve(a, b)
    bg = np.empty(n)
    bg[og] = b[oo]
    res = mg.solve(bg, precision=precision, rtol=1e-12, maxit=50)
    x = np.asarray(res[0] if isinstance(res, tuple) else res)
    assert np.abs(x[og] - want[oo]).max() <= 1e-8 * np.abs(want).max()
