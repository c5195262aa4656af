"""The element loop takes small meshes one element per thread and larger ones
by patches of families: meshes on both sides of each limit (FP32, FP64), plain
and Dirichlet, with hanging vertices on all sides and on the domain boundary,
against the oracle; and a mesh that keeps no node lists, which has families
only, against one that does.

Tolerances as for the families: 1e-12 of the largest entry in FP64, 1e-6 of the
norm in FP32 (sums of at most a few hundred terms, each off by a dozen
roundings)."""
import numpy as np
import pytest

from dendro_gb300 import DA, MultiGrid, Octree, balanceOctree, datagen, points2Octree
from .test_gpu_families import DEPTH, _perm, _tree

pytestmark = pytest.mark.gpu


# 7 split + 8^level elements: the ends of a patch (families of the packed mesh), 31,970
# and 32,005 (around FP64's limit), 89,993 and 90,007 (around FP32's), 172,768 (patches)
@pytest.mark.parametrize("level,split", [(0, 0), (1, 1), (3, 0), (3, 63), (3, 64), (3, 65), (3, 193), (4, 3982), (4, 3987), (5, 8175), (5, 8177), (5, 20000)])
def test_both_sides_of_the_limits(ctx, oracle, level, split):
    octs = _tree(level, split, seed=split)
    bal = Octree.from_numpy(octs, DEPTH, ctx=ctx)
    da, oda = DA(bal), oracle.DA(octs, DEPTH)
    p = _perm(da.download()["node_xyz"], oda.node_xyz)
    x = np.random.Generator(np.random.PCG64(3)).uniform(-1, 1, oda.n_node)
    xg = np.empty_like(x)
    xg[p] = x
    packed = DA(bal, compressLut=True)
    for lap, mass in ((1.0, 1.0), (-2.5, 30.0)):
        want = oda.matvec(x, lap, mass)
        for d in (da, packed):
            got = d.matvec(xg, lapFac=lap, massFac=mass)[p]
            assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
            got = d.matvec(xg.astype(np.float32), precision=32, lapFac=lap, massFac=mass)[p]
            assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)
    mg, want = MultiGrid(bal), oda.dirichlet_matvec(x)
    assert np.abs(mg.matvec(0, xg)[p] - want).max() <= 1e-12 * np.abs(want).max()
    got = mg.matvec(0, xg.astype(np.float32), precision=32)[p]
    assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)


def test_blocks_that_take_several_patches(ctx, oracle):
    """More patches than blocks fit the chip (a patch is 128 families): the
    copies ahead run from patch to patch, over the last one's end."""
    rng = np.random.Generator(np.random.PCG64(4))
    bal = balanceOctree(points2Octree(datagen.mixture(400_000, rng), ctx=ctx))
    da, oda = DA(bal), oracle.DA(bal.to_numpy(), DEPTH)
    assert da.n_elem > 7 * 128 * 1500
    p = _perm(da.download()["node_xyz"], oda.node_xyz)
    x = rng.uniform(-1, 1, oda.n_node)
    xg = np.empty_like(x)
    xg[p] = x
    mg = MultiGrid(bal)
    for want, apply in ((oda.matvec(x), lambda v, q: da.matvec(v, precision=q)),
                        (oda.dirichlet_matvec(x), lambda v, q: mg.matvec(0, v, precision=q))):
        assert np.abs(apply(xg, 64)[p] - want).max() <= 1e-12 * np.abs(want).max()
        assert np.linalg.norm(apply(xg.astype(np.float32), 32)[p] - want) <= 1e-6 * np.linalg.norm(want)
