"""The element loop on FP64 vectors: 64-bit fixed point with an exponent per
family, floating point for patches whose values, factors or range do not allow
it.  Against the oracle's FP64 loop over everything the rule looks at: factors
of both signs and of any size, fields even and rough, with zeros, beyond the
exponents, not finite.

Tolerance: a family's result is off by a few 2^-57 of its largest value times
its row sums, the oracle's by some 2^-53 of that, and a row sums at most a few
hundred terms: 1e-13 of the largest entry where the field is of one scale."""
import numpy as np
import pytest

from dendro_gb300 import DA, MultiGrid, balanceOctree, datagen, points2Octree

pytestmark = pytest.mark.gpu
FACTORS = [(1.0, 1.0), (1.0, 0.0), (0.0, 1.0), (-3.7, 250.0), (1e-3, 1e6), (0.0, 0.0), (1e150, -1e150), (1e-140, 1e-140)]
FIELDS = ["uniform", "smooth", "node", "zeros", "large", "small", "window"]


@pytest.fixture(scope="module")
def mesh(ctx, oracle):
    rng = np.random.Generator(np.random.PCG64(31))
    p = np.concatenate([datagen.mixture(4000, rng), 0.5 + 1e-4 * rng.normal(size=(200, 3))])  # levels 2 to 16
    bal = balanceOctree(points2Octree(p, ctx=ctx))
    da, oda = DA(bal), oracle.DA(bal.to_numpy(), 30)
    xyz = da.download()["node_xyz"]
    og, oo = np.lexsort(xyz.T[::-1]), np.lexsort(oda.node_xyz.T[::-1])
    perm = np.empty(len(oo), np.int64)
    perm[oo] = og
    return bal, da, oda, perm


def _field(name, oda):
    rng = np.random.Generator(np.random.PCG64(32))
    n = oda.n_node
    u = rng.uniform(-1, 1, n)
    if name == "smooth":
        return np.sin(np.pi * (oda.node_xyz / 2.0**30)).prod(1) + 0.01
    if name == "node":
        return (np.arange(n) == n // 2) * 1.0
    if name == "zeros":
        return np.where(oda.node_xyz[:, 0] < 2**29, 0.0, u)
    scale = {"uniform": 1.0, "large": 1e250, "small": 1e-250, "window": 2.0**511}
    return u * scale[name]  # window: both sides of the largest exponent of the fixed form


@pytest.mark.parametrize("field", FIELDS)
def test_fields_and_factors(mesh, field):
    _, da, oda, perm = mesh
    x = _field(field, oda)
    xg = np.empty_like(x)
    xg[perm] = x
    for lap, mass in FACTORS:
        scale = np.abs(x).max() * max(abs(lap), abs(mass), 1e-300)
        if not 1e-280 < scale < 1e280:  # the results leave FP64 themselves
            continue
        want, got = oda.matvec(x, lap, mass), da.matvec(xg, lapFac=lap, massFac=mass)[perm]
        assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max(), (lap, mass)


def test_a_rough_field_keeps_every_scale(mesh, oracle):
    """Values over 400 decades: each row against the sum of the magnitudes of
    its own terms' families (elements within a parent's lattice reach)."""
    _, da, oda, perm = mesh
    rng = np.random.Generator(np.random.PCG64(33))
    x = rng.normal(size=oda.n_node) * 10.0 ** rng.uniform(-200, 200, oda.n_node)
    xg = np.empty_like(x)
    xg[perm] = x
    want, got = oda.matvec(x, 0.0, 1.0), da.matvec(xg, lapFac=0.0, massFac=1.0)[perm]
    h = 2.0 ** -oda.level.astype(float)
    top = np.abs(x)[oda.nodes].max(1) * h**3  # per element, then over the elements of a node, twice
    reach = np.zeros(oda.n_node)
    for _ in range(3):
        np.maximum.at(reach, oda.nodes.ravel(), np.repeat(top, 8))
        top = reach[oda.nodes].max(1)
    assert (np.abs(got - want) <= 1e-13 * reach).all()


@pytest.mark.parametrize("lap,mass", [(np.nan, 1.0), (1.0, np.inf), (1e300, 1e300)])
def test_factors_out_of_range_give_what_floating_point_gives(mesh, lap, mass):
    _, da, oda, perm = mesh
    x = _field("uniform", oda)
    xg = np.empty_like(x)
    xg[perm] = x
    with np.errstate(all="ignore"):
        want = oda.matvec(x, lap, mass)
    got = da.matvec(xg, lapFac=lap, massFac=mass)[perm]
    if np.isfinite(want).all():
        assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
    else:
        assert not np.isfinite(got).any()


def test_the_two_fp64_precisions_agree(mesh):
    bal, _, oda, perm = mesh
    mg = MultiGrid(bal)
    x = np.random.Generator(np.random.PCG64(34)).uniform(-1, 1, oda.n_node)
    a, b = mg.matvec(0, x, precision=64), mg.matvec(0, x, precision=48)
    assert np.abs(a - b).max() <= 1e-15 * np.abs(a).max()
