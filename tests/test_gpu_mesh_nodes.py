"""The mesh's families come from the octree's internal octants, which it
carries when it was built here and which are recovered from its leaves when it
came from records: both give the same mesh.  Records that are no complete
octree in order go element by element: a mesh if every vertex has an owner,
refused otherwise."""
import numpy as np
import pytest

from dendro_gb300 import DA, DendroError, Octree, balanceOctree, datagen, points2Octree

pytestmark = pytest.mark.gpu
DEPTH = 30


def _points(kind):
    rng = np.random.Generator(np.random.PCG64(17))
    if kind == "one point":
        return np.array([[0.2, 0.7, 0.9]])
    p = datagen.mixture(3000, rng)
    if kind == "deepest":  # leaves of level 30: 128-bit keys of the internal octants
        p[1] = p[0] + 2.0**-29
    if kind == "corner":
        p = np.concatenate([p, 1.0 - 2.0 ** -np.arange(3.0, 20.0)[:, None] * np.ones(3)])
    return p


@pytest.mark.parametrize("kind", ["one point", "mixture", "corner", "deepest"])
def test_mesh_of_records_is_the_mesh_of_the_built_octree(ctx, oracle, kind):
    bal = balanceOctree(points2Octree(_points(kind), ctx=ctx))
    rec = bal.to_numpy()
    a, b = DA(bal), DA(Octree.from_numpy(rec, DEPTH, ctx=ctx))
    da, db = a.download(), b.download()
    for k in da:
        assert np.array_equal(da[k], db[k]), k
    oda = oracle.DA(rec, DEPTH)
    assert a.n_node == oda.n_node
    x = np.random.Generator(np.random.PCG64(2)).uniform(-1, 1, a.n_node)
    # one rounding of each of at most a few hundred terms in another order
    assert np.abs(a.matvec(x) - b.matvec(x)).max() <= 1e-12 * np.abs(a.matvec(x)).max()


@pytest.mark.parametrize("kind", ["mixture", "deepest"])
def test_a_leaf_that_owns_no_node_may_be_missing(ctx, kind):
    bal = balanceOctree(points2Octree(_points(kind), ctx=ctx))
    rec, whole = bal.to_numpy(), DA(bal)
    d = whole.download()
    # a finest leaf (it hangs nobody's vertices) whose anchor hangs, off the positive boundary
    side = np.uint32(1) << (DEPTH - rec[:, 3])
    inner = (rec[:, :3] + side[:, None] < 1 << DEPTH).all(1)
    own_none = np.flatnonzero((d["hmask"] & 1 == 1) & (rec[:, 3] == rec[:, 3].max()) & inner)
    assert len(own_none)
    i = int(own_none[len(own_none) // 2])
    part = DA(Octree.from_numpy(np.delete(rec, i, axis=0), DEPTH, ctx=ctx))
    p = part.download()
    for k in d:
        assert np.array_equal(p[k], d[k] if k == "node_xyz" else np.delete(d[k], i, axis=0)), k
    x = np.random.Generator(np.random.PCG64(3)).uniform(-1, 1, whole.n_node)
    coef = np.ones((whole.n_elem, 2))
    coef[i] = 0.0
    want = whole.matvec_coef(coef, x)
    # one rounding of each of at most a few hundred terms in another order
    assert np.abs(part.matvec(x) - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("fault", ["owner missing", "last missing", "far apart", "level off", "unbalanced"])
def test_records_that_are_no_mesh_are_refused(ctx, fault):
    bal = balanceOctree(points2Octree(_points("mixture"), ctx=ctx))
    rec, i = bal.to_numpy(), 0
    if fault == "owner missing":
        i = int(np.flatnonzero(DA(bal).download()["hmask"] & 1 == 0)[40])
        rec = np.delete(rec, i, axis=0)
    elif fault == "last missing":
        rec = rec[:-1]
    elif fault == "far apart":
        rec = rec[::-1].copy()
    elif fault == "level off":
        rec[len(rec) // 2, 3] += 1
    else:  # the finest leaf three levels deeper at its first child
        j = int(np.argmax(rec[:, 3]))
        x, y, z, l = (int(v) for v in rec[j])
        deeper = []
        for q in range(l + 1, l + 4):
            h = 1 << (DEPTH - q)
            deeper.append([[x + (c & 1) * h, y + (c >> 1 & 1) * h, z + (c >> 2) * h, q] for c in range(8)])
        leaves = deeper[2] + deeper[1][1:] + deeper[0][1:]
        rec = np.concatenate([rec[:j], np.array(leaves, np.uint32), rec[j + 1:]])
    with pytest.raises(DendroError):
        DA(Octree.from_numpy(rec, DEPTH, ctx=ctx))
