"""Construction, balance and coarsening where their paths part: points whose
leading bits agree in long runs (all bits sorted), coordinates at the edges of
cells and of FP64 with extents that are powers of two (integer scaling) and not
(division), a balance whose list of new nodes overflows and starts again, and
octrees with and without their internal octants.  Against the oracle; whole
numbers, so equality."""
import numpy as np
import pytest

from dendro_gb300 import DendroError, Octree, balanceOctree, coarsenOctree, datagen, points2Octree, sortUniquePoints

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("run", [30, 32, 33, 200, 3000])
@pytest.mark.parametrize("n", [4000, 300_000])  # without and with the read-back of the bits that vary
def test_runs_of_equal_prefixes(ctx, oracle, run, n):
    rng = np.random.Generator(np.random.PCG64(run))
    p = datagen.gaussian(n, 0.5, 0.15, seed=run)
    at = rng.permutation(64**3)[:run]  # distinct cells of depth 30 in one cell of depth 24
    cell = 0.25 + 2.0**-30 * np.stack([at % 64, at // 64 % 64, at // 4096], 1)
    p[:run] = cell
    assert np.array_equal(points2Octree(p, ctx=ctx).to_numpy(), oracle.points_to_octree(p, 30, 1))


@pytest.mark.parametrize("glens", [(1.0, 1.0, 1.0), (2.0, 0.5, 4.0), (2.0**40, 2.0**-40, 1.0), (3.0, 1.0, 0.7)])
@pytest.mark.parametrize("depth", [30, 7])
def test_coordinates_at_edges(ctx, oracle, glens, depth):
    rng = np.random.Generator(np.random.PCG64(5))
    h = 2.0**-depth
    cell = rng.integers(0, 1 << depth, (400, 3)) * h
    eps = np.array([0.0, 2.0**-53, -(2.0**-53), 2.0**-54, h / 2, h * (1 - 2.0**-40)])
    u = np.clip((cell[:, None] + eps[None, :, None]).reshape(-1, 3), 0.0, 1.0 - 2.0**-53)
    u[:8] = np.array([0.0, -0.0, 5e-324, 2.0**-1022, 2.0**-60, h, 1.0 - 2.0**-53, 1.0 - h])[:, None]
    p = u * np.asarray(glens)
    want = oracle.quantize_sort(p, depth, glens)
    got = sortUniquePoints(p, gLens=glens, maxDepth=depth, ctx=ctx)
    want = np.asarray(want).reshape(-1, 4)
    first = np.r_[True, (want[1:] != want[:-1]).any(1)]
    assert np.array_equal(got, want[first])


@pytest.mark.parametrize("bad", [(1.0 + 1e-9, 0.5, 0.5), (-1e-9, 0.5, 0.5), (np.nan, 0.5, 0.5), (np.inf, 0.5, 0.5)])
@pytest.mark.parametrize("g", [1.0, 1.5])
def test_points_outside_are_refused_alike(ctx, bad, g):
    p = datagen.gaussian(1000, 0.5, 0.1, seed=3)
    p[500] = np.asarray(bad)
    p *= g
    with pytest.raises(DendroError) as e:
        points2Octree(p, gLens=(g, g, g), ctx=ctx)
    assert e.value.status == 4  # DG_ERR_DOMAIN


def test_a_balance_that_starts_again(ctx, oracle):
    """Isolated pairs of near points: paths of 27 levels, whose balance adds
    more nodes than the first list holds."""
    rng = np.random.Generator(np.random.PCG64(6))
    a = rng.integers(0, 1 << 12, (900, 3)) / 2.0**12 + 2.0**-14
    p = np.unique(np.concatenate([a, a + 2.0**-28 * np.array([1.0, 0.0, 0.0])]), axis=0)
    lin = points2Octree(p, ctx=ctx)
    ctx.profile(True)
    bal = balanceOctree(lin)
    starts = ctx.profile_stats()["bal_start"][1]
    ctx.profile(False)
    assert starts >= 2
    rec = lin.to_numpy()
    assert np.array_equal(bal.to_numpy(), oracle.balance(rec, 30))
    assert np.array_equal(balanceOctree(Octree.from_numpy(rec, 30, ctx=ctx)).to_numpy(), bal.to_numpy())


@pytest.mark.parametrize("kind", ["mixture", "deep", "one"])
def test_coarsening_and_balance_with_and_without_nodes(ctx, oracle, kind):
    p = datagen.gaussian(3000, 0.5, 0.2, seed=9) if kind != "one" else np.array([[0.2, 0.3, 0.4]])
    if kind == "deep":
        p[1] = p[0] + 2.0**-28
    o = balanceOctree(points2Octree(p, ctx=ctx))
    for _ in range(4):
        rec = o.to_numpy()
        plain = Octree.from_numpy(rec, 30, ctx=ctx)
        c = coarsenOctree(o)
        assert np.array_equal(c.to_numpy(), oracle.coarsen(rec, 30))
        assert np.array_equal(coarsenOctree(plain).to_numpy(), c.to_numpy())
        for corner in (True, False):
            want = oracle.balance(c.to_numpy(), 30, corner)
            assert np.array_equal(balanceOctree(c, incCorner=corner).to_numpy(), want)
            back = Octree.from_numpy(c.to_numpy(), 30, ctx=ctx)
            assert np.array_equal(balanceOctree(back, incCorner=corner).to_numpy(), want)
        o = balanceOctree(c)
