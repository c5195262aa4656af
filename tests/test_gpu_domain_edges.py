"""Clouds that lie on an edge or a face of the domain: their octrees' internal
octants have two or four of the eight child numbers only, the nodes' hash table
must serve them all the same.  Mesh, element loop and solve against the oracle
(tolerances as for the other clouds: 1e-12 of the largest entry; the residual of
a solution to 1e-8 checked with the oracle's operator)."""
import numpy as np
import pytest

from dendro_gb300 import DA, MultiGrid, balanceOctree, points2Octree

pytestmark = pytest.mark.gpu


def _cloud(kind, n):
    rng = np.random.Generator(np.random.PCG64(n))
    if kind == "diagonal":
        return np.repeat(rng.random((n, 1)), 3, axis=1)
    p = rng.random((n, 3))
    fixed = {"edge": (0, 1), "top edge": (1, 2), "face": (2,), "top face": (0,)}[kind]
    for a in fixed:
        p[:, a] = 1.0 - 2.0**-30 if kind.startswith("top") else 0.0
    return p


@pytest.mark.parametrize("kind,n", [("edge", 300), ("edge", 1000), ("edge", 5000), ("top edge", 2000),
                                    ("face", 2000), ("face", 28000), ("face", 28600), ("top face", 28300),
                                    ("diagonal", 500)])
def test_mesh_and_solve(ctx, oracle, kind, n):
    p = _cloud(kind, n)
    lin = points2Octree(p, ctx=ctx)
    bal = balanceOctree(lin)
    rec = bal.to_numpy()
    assert np.array_equal(rec, oracle.balance(oracle.points_to_octree(p, 30, 1), 30))
    da, oda = DA(bal), oracle.DA(rec, 30)
    xyz = da.download()["node_xyz"]
    og, oo = np.lexsort(xyz.T[::-1]), np.lexsort(oda.node_xyz.T[::-1])
    assert np.array_equal(xyz[og], oda.node_xyz[oo])
    x = np.random.Generator(np.random.PCG64(1)).uniform(-1, 1, oda.n_node)
    xg = np.empty_like(x)
    xg[og] = x[oo]
    want = oda.matvec(x)
    assert np.abs(da.matvec(xg)[og] - want[oo]).max() <= 1e-12 * np.abs(want).max()
    mg = MultiGrid(bal)
    b = np.where(oda.bdy(), 0.0, oda.matvec(np.ones(oda.n_node), 0.0, 1.0))
    bg = np.empty_like(b)
    bg[og] = b[oo]
    sol, _, _ = mg.solve(bg, precision=64, rtol=1e-8, maxit=100)
    u = np.empty_like(b)
    u[oo] = sol[og]
    assert np.linalg.norm(b - oda.dirichlet_matvec(u)) <= 2e-8 * np.linalg.norm(b)
