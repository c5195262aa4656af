"""Every row of the element loop is as exact as its own terms allow, however
large the values beside it: fields of one node, that fall by a factor of 10 per
element, over many decades and zero on one side, on meshes that go element by
element and on meshes (and packed ones) that go by families.

Bound of row i: u B_i times a count of roundings, with u the unit roundoff and
B = sum over the elements of |P^T| (2 |lap| |K| + 7 |mass| M) |P| |x|, P the
hanging vertices' interpolation; the factors cover how a loop splits an entry
into sums and differences within a vertex's class and to its opposite (opposite
3/27 + 4/27 where M has 1/27).  Roundings: interpolation and its transpose 6, sums
and differences of a class 5, its products 3, a row 4, the 8 elements of a family 8,
the families of a node 8, factors 4: 38, and as many in the FP64 reference: 64 in
FP32, 96 in FP64.

Smooth fields: the rows of K sum to 0, and a row is as exact as the differences
between its vertices allow, B = sum of |P^T| (2 |lap| |K_ij| |x_j - x_i| + 7 |mass|
M |x|), to which hanging vertices, whose values are rounded, add themselves.

FP64 by families runs in fixed point: the values are cut at U = 2^-54 of the
family's largest, which a row's terms (2 (lap + mass) U with the roundings) feel by
at most 2^5 (classes of vertices reach 2^-5 of the largest) times 6 / 2: 96 u of
the bound, and 256 with both.

The reference is the dense form in FP64 with the matrices' zeros as zeros (the
oracle's stencil tables hold 1e-17 in their place where the compiler contracts
multiplications and additions)."""
import numpy as np
import pytest

from dendro_gb300 import DA, MultiGrid, Octree, balanceOctree, datagen, points2Octree

from .test_gpu_families import DEPTH, _perm, _tree

pytestmark = pytest.mark.gpu

# trilinear stiffness and mass on [-1, 1]^3 by the number of axes on which two vertices differ
_STEPS = np.array([[bin(i ^ j).count("1") for j in range(8)] for i in range(8)])
_K = np.array([2.0 / 3.0, 0.0, -1.0 / 6.0, -1.0 / 6.0])[_STEPS]
_M = np.array([8.0, 4.0, 2.0, 1.0])[_STEPS] / 27.0


class Dense:
    """The operator (apply) and B (bound), with per-element factors lap, mass
    (scalars or arrays)."""

    def __init__(self, oda):
        self.oda, self.groups = oda, []
        kind = oda.child.astype(np.int64) << 8 | oda.hmask
        for g in np.unique(kind):
            c, hm = int(g) >> 8, int(g) & 255
            p = np.zeros((8, 8))
            for k in range(8):
                subs = [s for s in range(8) if s & (k ^ c) == s] if hm >> k & 1 else None
                for s in subs or [k ^ c]:
                    p[k, c ^ s] += 1.0 / len(subs or [0])
            self.groups.append((np.flatnonzero(kind == g), p))

    def _sum(self, x, k, m, lap, mass):
        d = self.oda
        lap, mass = (np.broadcast_to(f, d.n_elem) for f in (lap, mass))
        h = 2.0 ** -d.level.astype(float)
        y = np.zeros(d.n_node)
        for e, p in self.groups:
            a = x[d.nodes[e]] @ p.T
            r = (a @ k) * (lap[e] * h[e] / 2)[:, None] + (a @ m) * (mass[e] * h[e] ** 3 / 8)[:, None]
            np.add.at(y, d.nodes[e].ravel(), (r @ p).ravel())
        return y

    def apply(self, x, lap=1.0, mass=1.0):
        return self._sum(x, _K, _M, lap, mass)

    def exact(self, x):
        """K x + M x in extended precision"""
        d, ld = self.oda, np.longdouble
        k = np.array([ld(2) / 3, ld(0), -ld(1) / 6, -ld(1) / 6])[_STEPS]
        m = np.array([8, 4, 2, 1], ld)[_STEPS] / ld(27)
        h = (2.0 ** -d.level.astype(float)).astype(ld)
        y = np.zeros(d.n_node, ld)
        for e, p in self.groups:
            a = x.astype(ld)[d.nodes[e]] @ p.T.astype(ld)
            r = (a @ k) * (h[e] / 2)[:, None] + (a @ m) * (h[e] ** 3 / 8)[:, None]
            np.add.at(y, d.nodes[e].ravel(), (r @ p.astype(ld)).ravel())
        return y

    def bound(self, x, lap=1.0, mass=1.0):
        return self._sum(np.abs(x), 2 * np.abs(_K), 7 * _M, np.abs(lap), np.abs(mass))

    def smooth_bound(self, x, lap=1.0, mass=1.0):
        d = self.oda
        y = self._sum(np.abs(x), 0 * _K, 7 * _M, 0.0, abs(mass))
        for e, p in self.groups:
            a = x[d.nodes[e]] @ p.T
            held = np.abs(a) * ((p != 0).sum(1) > 1)  # hanging
            diff = np.abs(a[:, None, :] - a[:, :, None]) + held[:, None, :] + held[:, :, None]
            r = np.einsum("ij,eij->ei", 2 * np.abs(_K), diff) * (abs(lap) * 2.0 ** -d.level[e].astype(float) / 2)[:, None]
            np.add.at(y, d.nodes[e].ravel(), (r @ np.abs(p)).ravel())
        return y

    def dirichlet(self, x):
        """... with boundary rows the identity and boundary columns dropped"""
        edge = self.oda.bdy()
        inner = np.where(edge, 0.0, x)
        return np.where(edge, x, self.apply(inner)), np.where(edge, 0.0, self.bound(inner))


@pytest.fixture(scope="module", params=["elements", "families", "packed"])
def mesh(request, ctx, oracle):
    rng = np.random.Generator(np.random.PCG64(41))
    if request.param == "families":  # above both limits
        bal = balanceOctree(points2Octree(datagen.mixture(20_000, rng), ctx=ctx))
    else:
        bal = Octree.from_numpy(_tree(4, 700, seed=3), DEPTH, ctx=ctx)
    da, oda = DA(bal, compressLut=request.param == "packed"), oracle.DA(bal.to_numpy(), DEPTH)
    assert (da.n_elem > 90_000) if request.param == "families" else (da.n_elem < 32_000)
    return bal, da, oda, _perm(da.download()["node_xyz"], oda.node_xyz), Dense(oda)


FIELDS = ["node", "decay", "decades", "half", "mixed"]


def _field(name, oda):
    rng = np.random.Generator(np.random.PCG64(42))
    n = oda.n_node
    u = rng.uniform(-1, 1, n)
    at = oda.node_xyz / 2.0**DEPTH
    size = np.zeros(n)  # of the elements at a node
    np.maximum.at(size, oda.nodes.ravel(), np.repeat(2.0 ** -oda.level.astype(float), 8))
    if name == "node":
        return (np.arange(n) == n // 2) * 1.0
    if name == "decay":
        return 10.0 ** -np.minimum(np.abs(at - 0.43).max(1) / np.median(size), 12.0)
    if name == "decades":
        return u * 10.0 ** rng.uniform(-8, 8, n)
    if name == "half":
        return np.where(at[:, 0] < 0.5, 0.0, u)
    return np.where(rng.random(n) < 0.02, u * 1e9, u)


def _check(got, want, bound, roundings, unit):
    assert (np.abs(got - want) <= roundings * unit * bound).all()


def _put(x, p):
    xg = np.empty_like(x)
    xg[p] = x
    return xg


@pytest.mark.parametrize("field", FIELDS)
def test_single_precision(mesh, field):
    bal, da, oda, p, dense = mesh
    x = _field(field, oda).astype(np.float32)
    x64 = x.astype(np.float64)
    for lap, mass in ((1.0, 1.0), (1.0, 0.0), (0.0, 1.0), (-3.0, 40.0)):
        got = da.matvec(_put(x, p), precision=32, lapFac=lap, massFac=mass)[p]
        _check(got, dense.apply(x64, lap, mass), dense.bound(x64, lap, mass), 64, 2.0**-24)
    if not da.compressLut:
        got = MultiGrid(bal).matvec(0, _put(x, p), precision=32)[p]
        _check(got, *dense.dirichlet(x64), 64, 2.0**-24)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("field", FIELDS)
def test_factors_per_element(mesh, field, precision):
    _, da, oda, p, dense = mesh
    t = np.float32 if precision == 32 else np.float64
    x = _field(field, oda).astype(t)
    coef = np.random.Generator(np.random.PCG64(43)).uniform(0.05, 4.0, (da.n_elem, 2))
    got = da.matvec_coef(coef, _put(x, p), precision=precision)[p]
    x64 = x.astype(np.float64)
    f = coef[:, 0], coef[:, 1]
    _check(got, dense.apply(x64, *f), dense.bound(x64, *f), 64 if precision == 32 else 96, 2.0**-24 if precision == 32 else 2.0**-53)


@pytest.mark.parametrize("precision", [32, 64])
def test_largest_values(mesh, precision):
    """Values at the end of the range, of both signs: the rows, which are far
    smaller, are finite."""
    _, da, oda, p, dense = mesh
    t = np.float32 if precision == 32 else np.float64
    u = np.random.Generator(np.random.PCG64(44)).choice([-1.0, 1.0], oda.n_node)
    x = (u * 0.99 * np.finfo(t).max).astype(t)
    got = da.matvec(_put(x, p), precision=precision)[p].astype(np.float64)
    scale = 2.0 ** (-120 if precision == 32 else -1000)  # exact; the reference's sums may not overflow either
    x64 = x.astype(np.float64) * scale
    _check(got * scale, dense.apply(x64), dense.bound(x64), 64 if precision == 32 else 96, 2.0**-24 if precision == 32 else 2.0**-53)


@pytest.mark.parametrize("field", FIELDS)
def test_double_precision_element_by_element(mesh, field):
    bal, da, oda, p, dense = mesh
    if da.compressLut or da.n_elem > 32_000:
        pytest.skip("goes by families")
    x = _field(field, oda)
    for lap, mass in ((1.0, 1.0), (1.0, 0.0), (0.0, 1.0), (-3.0, 40.0)):
        _check(da.matvec(_put(x, p), lapFac=lap, massFac=mass)[p], dense.apply(x, lap, mass), dense.bound(x, lap, mass), 96, 2.0**-53)
    _check(MultiGrid(bal).matvec(0, _put(x, p))[p], *dense.dirichlet(x), 96, 2.0**-53)


@pytest.mark.parametrize("field", FIELDS)
def test_double_precision_by_families(mesh, field):
    bal, da, oda, p, dense = mesh
    if not da.compressLut and da.n_elem < 32_000:
        pytest.skip("goes element by element")
    x = _field(field, oda)
    for lap, mass in ((1.0, 1.0), (1.0, 0.0), (0.0, 1.0), (-3.0, 40.0)):
        _check(da.matvec(_put(x, p), lapFac=lap, massFac=mass)[p], dense.apply(x, lap, mass), dense.bound(x, lap, mass), 256, 2.0**-53)
    if not da.compressLut:
        _check(MultiGrid(bal).matvec(0, _put(x, p))[p], *dense.dirichlet(x), 256, 2.0**-53)


@pytest.mark.parametrize("field", ["constant", "linear", "sines"])
def test_smooth_fields(mesh, field):
    _, da, oda, p, dense = mesh
    at = oda.node_xyz / 2.0**DEPTH
    x = {"constant": np.full(oda.n_node, 0.7), "linear": 1.0 + at @ np.array([0.5, -0.25, 2.0]),
         "sines": 1.5 + np.sin(np.pi * at).prod(1)}[field]
    one = np.ones((da.n_elem, 2))
    for t, roundings, unit in ((np.float32, 64, 2.0**-24), (np.float64, 96, 2.0**-53)):
        xt = x.astype(t)
        x64, prec = xt.astype(np.float64), 32 if t is np.float32 else 64
        if prec == 64 and da.n_elem > 32_000:
            continue  # by families in fixed point; extended precision takes long
        want, bound = dense.apply(x64) if prec == 32 else dense.exact(x64), dense.smooth_bound(x64)
        loops = [da.matvec_coef(one, _put(xt, p), precision=prec)[p]]
        if prec == 32 or not da.compressLut:
            loops.append(da.matvec(_put(xt, p), precision=prec)[p])
        for got in loops:
            assert (np.abs(got - want) <= roundings * unit * bound).all()
