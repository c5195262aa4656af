"""The element loops by families on meshes above the sizes that go element by
element (90,000 elements in FP32, 32,000 in FP64) and on packed meshes, which
always go by families: last patches one family short, full and one over (a patch
is 128 families), the Dirichlet form, values that are not finite, and the
fixed-point form against its own range, factors and an independent FP64 loop.

Tolerances as for the families: 1e-12 of the largest entry in FP64, 1e-6 of the
norm in FP32; the fixed form 1e-13 of the largest entry."""
import numpy as np
import pytest

from dendro_gb300 import DA, MultiGrid, Octree, balanceOctree, datagen, points2Octree

from .test_gpu_families import DEPTH, _perm, _tree
from .test_gpu_fixed_point import FACTORS, FIELDS, _field
from .test_gpu_row_accuracy import Dense

pytestmark = pytest.mark.gpu


def _put(x, p):
    xg = np.empty_like(x)
    xg[p] = x
    return xg


# 8^5 + 7 split elements in 4,096 + split families (32 patches and split / 128)
@pytest.mark.parametrize("split", [8192 + 127, 8192 + 128, 8192 + 129])
def test_last_patches(ctx, oracle, split):
    octs = _tree(5, split, seed=split)
    bal = Octree.from_numpy(octs, DEPTH, ctx=ctx)
    da, oda = DA(bal), oracle.DA(octs, DEPTH)
    assert da.n_elem > 90_000
    p = _perm(da.download()["node_xyz"], oda.node_xyz)
    x = np.random.Generator(np.random.PCG64(51)).uniform(-1, 1, oda.n_node)
    mg = MultiGrid(bal)
    for want, apply in ((oda.matvec(x), lambda v, q: da.matvec(v, precision=q)),
                        (oda.dirichlet_matvec(x), lambda v, q: mg.matvec(0, v, precision=q))):
        got = apply(_put(x.astype(np.float32), p), 32)[p]
        assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)
        for scale in (1.0, 1e-300, 1e300):  # fixed point, and floating point below and above its range
            got = apply(_put(x * scale, p), 64)[p] / scale
            assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


@pytest.fixture(scope="module")
def mesh(ctx, oracle):
    rng = np.random.Generator(np.random.PCG64(52))
    pts = np.concatenate([datagen.mixture(20_000, rng), 0.5 + 1e-4 * rng.normal(size=(400, 3))])
    bal = balanceOctree(points2Octree(pts, ctx=ctx))
    da, oda = DA(bal), oracle.DA(bal.to_numpy(), DEPTH)
    assert da.n_elem > 100_000
    return bal, da, oda, _perm(da.download()["node_xyz"], oda.node_xyz)


@pytest.mark.parametrize("kind", ["mesh", "packed", "factors", "dirichlet"])
@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_values_that_are_not_finite(ctx, oracle, mesh, kind, precision, value):
    """They reach the rows of the elements that hold them, and no other."""
    if kind in ("mesh", "dirichlet"):
        bal, da, oda, p = mesh
    else:
        octs = _tree(3, 65, seed=5)
        bal, oda = Octree.from_numpy(octs, DEPTH, ctx=ctx), oracle.DA(octs, DEPTH)
        da = DA(bal, compressLut=kind == "packed")
        p = _perm(da.download()["node_xyz"], oda.node_xyz)
    mg = MultiGrid(bal) if kind == "dirichlet" else None
    coef = np.random.Generator(np.random.PCG64(53)).uniform(0.5, 2.0, (da.n_elem, 2))
    edge = oda.bdy()
    for node in (0, oda.n_node // 3, oda.n_node // 2, oda.n_node - 1):
        x = np.random.Generator(np.random.PCG64(node)).uniform(-1, 1, oda.n_node)
        x[node] = value
        x = x.astype(np.float32 if precision == 32 else np.float64)
        rows = np.zeros(oda.n_node, bool)
        rows[oda.nodes[(oda.nodes == node).any(1)].ravel()] = True
        if kind == "dirichlet":
            rows &= ~edge & ~edge[node]
            rows[node] = True
            got = mg.matvec(0, _put(x, p), precision=precision)[p]
        elif kind == "factors":
            got = da.matvec_coef(coef, _put(x, p), precision=precision)[p]
        else:
            got = da.matvec(_put(x, p), precision=precision)[p]
        assert np.array_equal(~np.isfinite(got), rows)


@pytest.mark.parametrize("field", FIELDS)
def test_fixed_point_fields_and_factors(mesh, field):
    _, da, oda, p = mesh
    x = _field(field, oda)
    for lap, mass in FACTORS:
        with np.errstate(over="ignore"):
            scale = np.abs(x).max() * max(abs(lap), abs(mass), 1e-300)
        if not 1e-280 < scale < 1e280:  # the results leave FP64 themselves
            continue
        want, got = oda.matvec(x, lap, mass), da.matvec(_put(x, p), lapFac=lap, massFac=mass)[p]
        assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max(), (lap, mass)


def test_fixed_point_against_floating_point(mesh):
    """The loop with factors per element is FP64 throughout."""
    _, da, oda, p = mesh
    x = np.random.Generator(np.random.PCG64(54)).uniform(-1, 1, oda.n_node)
    for lap, mass in ((1.0, 1.0), (2.0, -300.0)):
        a = da.matvec(x, lapFac=lap, massFac=mass)
        b = da.matvec_coef(np.tile([lap, mass], (da.n_elem, 1)), x)
        assert np.abs(a - b).max() <= 1e-14 * np.abs(b).max()
        assert not np.array_equal(a, b)  # they are two loops


def test_many_families_go_alone(mesh):
    """Large values at some of the nodes, so that patches hold families of uneven
    values, one to nearly all of them (bounds: test_gpu_row_accuracy)."""
    bal, da, oda, p = mesh
    dense, mg = Dense(oda), MultiGrid(bal)
    rng = np.random.Generator(np.random.PCG64(55))
    for share in (1e-4, 1e-3, 1e-2, 1e-1):
        x = rng.uniform(-1, 1, oda.n_node) * np.where(rng.random(oda.n_node) < share, 1e12, 1.0)
        got = da.matvec(_put(x, p))[p]
        assert (np.abs(got - dense.apply(x)) <= 256 * 2.0**-53 * dense.bound(x)).all()
        got = mg.matvec(0, _put(x, p))[p]
        want, bound = dense.dirichlet(x)
        assert (np.abs(got - want) <= 256 * 2.0**-53 * bound).all()
