"""The balance checks the list of nodes that its hash table gave before it
returns an octree made from them: a node that stands twice, is missing above
another one, out of order or of no level is an error.  The rule, compiled for the
host, on the nodes of octrees (one cloud and two, 64- and 128-bit keys) and on
lists with one such fault."""
import os
import subprocess

import numpy as np
import pytest

from dendro_gb300 import build as cuda_build
from dendro_gb300 import datagen

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("node_order")
    exe = str(tmp / "node_order")
    cmd = [cuda_build.nvcc(), *cuda_build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-O1",
           "-I" + os.path.join(cuda_build.ROOT, "include"), os.path.join(HERE, "cpp", "node_order_main.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(keys, lm):
        path = str(tmp / "keys.bin")
        np.array([[k & (2**64 - 1), k >> 64] for k in keys], np.uint64).tofile(path)
        out = subprocess.run([exe, path, str(lm)], capture_output=True, text=True, check=True).stdout.split()
        assert len(set(out)) == 1  # both key widths agree
        return int(out[0])

    return run


def _nodes(octs, lm, cloud=0):
    """Keys of the internal octants, in preorder: path (3 bits per level to level
    lm, the cloud above) over 5 bits of level."""
    keys = set()
    for x, y, z, l in octs.tolist():
        for d in range(l):
            path = cloud
            for b in range(lm):
                c = 0
                if b < d:
                    s = 29 - b
                    c = (x >> s & 1) | (y >> s & 1) << 1 | (z >> s & 1) << 2
                path = path << 3 | c
            keys.add(path << 5 | d)
    return sorted(keys)


@pytest.mark.parametrize("deep", [False, True])
def test_rule(rule, oracle, deep):
    p = datagen.gaussian(150, 0.5, 0.2, seed=4)
    if deep:
        p[1] = p[0] + 2.0**-28
    octs = oracle.balance(oracle.points_to_octree(p, 30, 1), 30)
    lm = int(octs[:, 3].max()) - 1
    keys = _nodes(octs, lm)
    assert (keys[-1] >> 64 > 0) == deep
    assert 7 * len(keys) + 1 == len(octs)
    assert rule(keys, lm) == -1
    both = keys + _nodes(octs, lm, cloud=5)
    assert rule(both, lm) == -1
    n = len(keys)
    inner = [i for i in range(1, n - 1) if (keys[i + 1] & 31) > (keys[i] & 31)]  # nodes with nodes below them
    for i in inner[:: max(1, len(inner) // 20)]:
        assert rule(both[:i] + both[i + 1:], lm) == i, "a missing parent"
        assert rule(both[:i] + both[i:i + 1] + both[i:], lm) == i + 1, "twice"
        assert rule(both[:i] + [both[i + 1], both[i]] + both[i + 2:], lm) in (i, i + 1), "out of order"
        assert rule(both[:i] + [both[i] | 31] + both[i + 1:], lm) == i, "no level"
    assert rule(both[1:], lm) == 0, "no root"
    assert rule(both[:n] + both[n + 1:], lm) == n, "no root of the second cloud"
