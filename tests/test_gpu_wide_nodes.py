"""Batches whose internal octants need 128-bit keys (cloud index above deep
paths): the segmented construction and balance give every cloud the octree it
gets alone (64-bit keys), again and again."""
import numpy as np
import pytest

from dendro_gb300 import balanceOctree, datagen, points2Octree, points2OctreeBatch

pytestmark = pytest.mark.gpu


def test_wide_keys_repeat_the_single_cloud_octrees(ctx):
    # 300 clouds (9 index bits); two points 2^-19 apart make leaves of level 19
    # and deeper (3 * 18 + 9 + 5 > 64)
    rng = np.random.Generator(np.random.PCG64(91))
    sizes = datagen.cloud_sizes(300, 50, 3e4, seed=92)
    clouds = [datagen.mixture(int(n), rng) for n in sizes]
    for c in clouds[::7]:
        c[0] = np.array([0.3, 0.6, 0.7])
        c[1] = c[0] + 2.0**-19
    alone = []
    for c in clouds:
        bal = balanceOctree(points2Octree(c, ctx=ctx))
        alone.append(bal.to_numpy())
    lin = points2OctreeBatch(clouds, ctx=ctx)
    want = np.concatenate(alone)
    for _ in range(5):
        bal = balanceOctree(lin)
        assert np.array_equal(np.diff(bal.segments()), [len(a) for a in alone])
        assert np.array_equal(bal.to_numpy(), want)
        bal.free()
