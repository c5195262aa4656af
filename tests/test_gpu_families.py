"""The element loop by sibling families at the sizes where its patches end:
one element, one family, a patch of families less one, exactly full and one
more, families with subdivided children and with hanging points on every
side.  Against the oracle's element loop.

Tolerances.  FP64: a row sums at most a few hundred terms, each off by a dozen
roundings of 2^-53, so 1e-12 of the largest entry.  FP32: the same with 2^-24,
averaged over the vector: 1e-6 relative L2.  Fixed point: a family's results
are off by less than 2^-50 of its patch's largest row, so 1e-12 of the norm
for a field that is rough everywhere."""
import numpy as np
import pytest

from dendro_gb300 import DA, MultiGrid, Octree

pytestmark = pytest.mark.gpu
DEPTH = 30


def _perm(xyz_gpu, xyz_ref):
    og = np.lexsort(xyz_gpu.T[::-1])
    oo = np.lexsort(xyz_ref.T[::-1])
    assert np.array_equal(xyz_gpu[og], xyz_ref[oo])
    p = np.empty(len(oo), np.int64)
    p[oo] = og
    return p


def _tree(level, split, seed=0):
    """The uniform octree of a level with `split` of its leaves subdivided
    once (2:1 balanced: neighbours differ by one level), in Morton order."""
    n = 1 << level
    g = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)[:, ::-1].astype(np.uint64)
    rng = np.random.Generator(np.random.PCG64(seed))
    cut = np.zeros(len(g), bool)
    cut[rng.permutation(len(g))[:split]] = True
    bits = np.array([[k & 1, k >> 1 & 1, k >> 2] for k in range(8)], np.uint64)
    fine = (2 * g[cut][:, None] + bits).reshape(-1, 3) << np.uint64(DEPTH - level - 1)
    octs = np.concatenate([np.column_stack([g[~cut] << np.uint64(DEPTH - level), np.full((~cut).sum(), level, np.uint64)]),
                           np.column_stack([fine, np.full(len(fine), level + 1, np.uint64)])])
    key = np.zeros(len(octs), np.uint64)
    for b in range(5):  # levels up to 5 suffice here
        for a in range(3):
            key |= (octs[:, a] >> np.uint64(DEPTH - 1 - b) & np.uint64(1)) << np.uint64(3 * (20 - b) + a)
    return octs[np.argsort(key, kind="stable")].astype(np.uint32)


TREES = [(0, 0), (1, 0), (1, 1), (1, 7), (2, 0), (2, 13), (3, 0), (3, 63), (3, 64), (3, 65), (3, 192), (3, 193), (3, 500)]


@pytest.mark.parametrize("level,split", TREES)
def test_element_loops(ctx, oracle, level, split):
    octs = _tree(level, split, seed=split)
    bal = Octree.from_numpy(octs, DEPTH, ctx=ctx)
    da, oda = DA(bal), oracle.DA(octs, DEPTH)
    p = _perm(da.download()["node_xyz"], oda.node_xyz)
    rng = np.random.Generator(np.random.PCG64(1))
    x = rng.uniform(-1, 1, oda.n_node)
    xg = np.empty_like(x)
    xg[p] = x

    def close64(got, want):
        assert np.abs(got[p] - want).max() <= 1e-12 * np.abs(want).max()

    def close32(got, want):
        assert np.linalg.norm(got[p] - want) <= 1e-6 * np.linalg.norm(want)

    for lap, mass in ((1.0, 1.0), (0.0, 1.0), (2.5, 0.0)):
        want = oda.matvec(x, lap, mass)
        close64(da.matvec(xg, lapFac=lap, massFac=mass), want)
        close32(da.matvec(xg.astype(np.float32), precision=32, lapFac=lap, massFac=mass), want)
    coef = rng.uniform(0.05, 4.0, (da.n_elem, 2))
    want = oracle.matvec_coef(oda, coef, x)
    close64(da.matvec_coef(coef, xg), want)
    close32(da.matvec_coef(coef, xg.astype(np.float32), precision=32), want)
    packed = DA(bal, compressLut=True)
    assert np.array_equal(packed.download()["nodes"], da.download()["nodes"])
    close64(packed.matvec(xg), oda.matvec(x))
    mg = MultiGrid(bal, max_coarse_elems=len(octs))
    want = oda.dirichlet_matvec(x)
    close64(mg.matvec(0, xg), want)
    close32(mg.matvec(0, xg.astype(np.float32), precision=32), want)
    for scale in (1.0, 1e-300, 1e300):
        got = mg.matvec(0, xg * scale, precision=48)[p] / scale
        assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_non_finite_values_reach_their_elements_only(ctx, oracle, precision, value):
    """A non-finite x makes exactly the rows of the elements that hold the
    node non-finite."""
    octs = _tree(3, 65, seed=5)
    da, oda = DA(Octree.from_numpy(octs, DEPTH, ctx=ctx)), oracle.DA(octs, DEPTH)
    p = _perm(da.download()["node_xyz"], oda.node_xyz)
    for node in (0, oda.n_node // 3, oda.n_node // 2, oda.n_node - 1):
        x = np.random.Generator(np.random.PCG64(node)).uniform(-1, 1, oda.n_node)
        x[node] = value
        xg = np.empty_like(x)
        xg[p] = x
        held = np.zeros(oda.n_node, bool)
        held[oda.nodes[(oda.nodes == node).any(1)].ravel()] = True
        got = da.matvec(xg.astype(np.float32) if precision == 32 else xg, precision=precision)[p]
        assert np.array_equal(~np.isfinite(got), held)
