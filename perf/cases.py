"""The measured workloads: what users of this library have it do, through its Python API.

Sizes and distributions are those of the benchmark and the tests: Gaussian, log-normal and
Gaussian-mixture point clouds at maxDepth 30, one point per octant, requests of 1e4 to 8e6 points.

  build     points2Octree + balanceOctree, the records read into a device tensor
  batch     the same for many clouds in one segmented call
  mesh      ot::DA of a balanced octree and the first operator application on it
  apply     Laplacian + mass element loop on a DA that the program keeps
  request   one served request: cloud -> octree -> balance -> multigrid -> load vector -> solution
  solve     CG + V-cycle on a hierarchy that the program keeps
"""
import numpy as np
import torch

import dendro_gb300 as dg

DEPTH = 30
DEV = "cuda"


def listed():
    return [
        # the smallest clouds of the serving stream: launches and read-backs count
        {"name": "build_20k", "kind": "build", "cloud": "mixture", "n": 20011},
        # the plain-method cloud
        {"name": "build_1m", "kind": "build", "cloud": "gaussian", "n": 1000000},
        # a quarter of the scale workload: adaptive log-normal cloud, 9e7 balanced octants
        {"name": "build_16m", "kind": "build", "cloud": "lognormal", "n": 16000000},
        # a batch as the server forms it: clouds of mixed sizes in one segmented pass
        {"name": "batch_40", "kind": "batch", "clouds": 40, "lo": 10000, "hi": 400000},
        # set-up of a discretisation: mesh, then the operator once
        {"name": "mesh_1m", "kind": "mesh", "cloud": "gaussian", "n": 999983},
        # explicit steps and smoothers on a small mesh
        {"name": "apply32_20k", "kind": "apply", "cloud": "mixture", "n": 20011, "precision": 32},
        # the same on a mesh far larger than the caches
        {"name": "apply32_4m", "kind": "apply", "cloud": "lognormal", "n": 4000000, "precision": 32},
        # the reference's own precision
        {"name": "apply64_1m", "kind": "apply", "cloud": "gaussian", "n": 1000003, "precision": 64},
        # whole served requests, a small and a large one
        {"name": "request_20k", "kind": "request", "cloud": "mixture", "n": 20011},
        {"name": "request_1m", "kind": "request", "cloud": "lognormal", "n": 1200000},
        # repeated solves on one hierarchy: the precision workload's FP32 V-cycle, and all FP64
        {"name": "solve32_4m", "kind": "solve", "cloud": "gaussian", "n": 4000000, "precision": 32},
        {"name": "solve64_500k", "kind": "solve", "cloud": "gaussian", "n": 500009, "precision": 64},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["build", "batch", "mesh", "apply", "apply", "request", "solve"])
    if kind == "batch":
        hi = size(20000, 400000)
        return {"kind": kind, "clouds": rng.randint(2, 40), "lo": 10000, "hi": hi}
    case = {"kind": kind, "cloud": rng.choice(["mixture", "gaussian", "lognormal"])}
    case["n"] = size(10000, {"build": 16e6, "mesh": 2e6, "apply": 4e6, "request": 1.2e6, "solve": 1e6}[kind])
    if kind in ("apply", "solve"):
        case["precision"] = rng.choice([32, 64])
    return case


# ---- inputs -------------------------------------------------------------------------------------
def _points(cloud, n, gen):
    """n points of a named distribution in [0, 1)^3 (FP64, on the device)."""
    z = torch.randn((n, 3), dtype=torch.float64, device=DEV, generator=gen)
    if cloud == "lognormal":
        u = torch.exp(z)
        return torch.clamp(u / (1.0 + u), max=float(np.nextafter(1.0, 0.0)))
    if cloud == "gaussian":
        p = 0.5 + 0.1 * z
    else:  # 1 to 8 isotropic Gaussians of widths 0.01 to 0.2
        k = int(torch.randint(1, 9, (1,), device=DEV, generator=gen))
        centre = 0.1 + 0.8 * torch.rand((k, 3), dtype=torch.float64, device=DEV, generator=gen)
        sigma = 0.01 * 20.0 ** torch.rand((k, 1), dtype=torch.float64, device=DEV, generator=gen)
        which = torch.randint(0, k, (n,), device=DEV, generator=gen)
        p = centre[which] + sigma[which] * z
    again = torch.rand((n, 3), dtype=torch.float64, device=DEV, generator=gen)
    outside = ((p < 0.0) | (p >= 1.0)).any(1, keepdim=True)
    return torch.where(outside, again, p)


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _load(unit):
    """The source term at points of the unit cube: a few smooth bumps."""
    f = torch.zeros(unit.shape[0], dtype=torch.float64, device=unit.device)
    for a, c, s in ((1.3, (0.4, 0.6, 0.5), 0.11), (0.8, (0.7, 0.3, 0.4), 0.07), (1.9, (0.5, 0.5, 0.7), 0.14)):
        d = unit - torch.tensor(c, dtype=torch.float64, device=unit.device)
        f += a * torch.exp((d * d).sum(1) * (-0.5 / (s * s)))
    return f


def _unit(nodes):
    return nodes.to(torch.float64) / float(1 << DEPTH)


def _vector(n, precision, gen):
    x = 2.0 * torch.rand(n, dtype=torch.float64, device=DEV, generator=gen) - 1.0
    return x if precision == 64 else x.to(torch.float32)


# Results go into buffers that the program keeps: room for this many octants and nodes per point
# (what lies past a result's end stays 0).
ROOM_OCTANTS, ROOM_NODES = 10, 7


def _room(n, rows, columns=None, dtype=torch.float64):
    return torch.zeros((n * rows,) if columns is None else (n * rows, columns), dtype=dtype, device=DEV)


def _head(buffer, n):
    if n > len(buffer):
        raise RuntimeError("a result of %d entries where there is room for %d" % (n, len(buffer)))
    return buffer[:n]


def _octree(points):
    lin = dg.points2Octree(points, maxDepth=DEPTH)
    bal = dg.balanceOctree(lin)
    lin.free()
    return bal


def prepare(case, seed):
    gen = _generator(seed)
    if case["kind"] == "batch":
        rng = np.random.default_rng(seed)
        sizes = np.rint(case["lo"] * (case["hi"] / case["lo"]) ** rng.random(case["clouds"])).astype(np.int64)
        points = torch.cat([_points("mixture", int(n), gen) for n in sizes])
        start = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
        out = _room(case["clouds"] * case["hi"], ROOM_OCTANTS, 4, torch.int32)
        return {"kind": "batch", "points": points, "start": start, "out": out}
    points = _points(case["cloud"], case["n"], gen)
    state = {"kind": case["kind"], "points": points}
    if case["kind"] == "build":
        state["out"] = _room(case["n"], ROOM_OCTANTS, 4, torch.int32)
        return state
    precision = case.get("precision", 64)
    single = case["kind"] == "apply" and precision == 32
    state.update(precision=precision, out=_room(case["n"], ROOM_NODES, None, torch.float32 if single else torch.float64))
    if case["kind"] == "request":
        return state
    bal = _octree(points)
    if case["kind"] == "solve":
        mg = dg.MultiGrid(bal)
        state.update(mg=mg, b=mg.rhs(_load(_unit(mg.level_nodes(0, device=True)))))
        return state
    da = dg.DA(bal)
    state["x"] = _vector(da.n_node, precision, gen)
    state.update({"bal": bal} if case["kind"] == "mesh" else {"da": da})
    return state


# ---- one pass -----------------------------------------------------------------------------------
def run(state):
    kind, out = state["kind"], state["out"]
    if kind in ("build", "batch"):
        if kind == "build":
            lin = dg.points2Octree(state["points"], maxDepth=DEPTH)
        else:
            lin = dg.points2OctreeBatch(state["points"], maxDepth=DEPTH, seg_start=state["start"])
        bal = dg.balanceOctree(lin)
        bal.download_to(_head(out, len(bal)))
        starts = bal.segments().astype(np.int64)
        lin.free()
        bal.free()
        return [out, starts]
    if kind == "mesh":
        da = dg.DA(state["bal"])
        da.matvec(state["x"], out=_head(out, da.n_node), precision=64)
        da.free()
    elif kind == "apply":
        da = state["da"]
        da.matvec(state["x"], out=_head(out, da.n_node), precision=state["precision"])
    elif kind == "solve":
        mg = state["mg"]
        mg.solve(state["b"], precision=state["precision"], rtol=1e-8, maxit=50, x=_head(out, mg.sizes[0][1]))
    else:
        bal = _octree(state["points"])
        mg = dg.MultiGrid(bal)
        b = mg.rhs(_load(_unit(mg.level_nodes(0, device=True))))
        mg.solve(b, precision=32, rtol=1e-8, maxit=50, x=_head(out, len(b)))
        mg.free()
        bal.free()
    return out


# balanced octants per point and nodes per octant of these clouds, and CG iterations to 1e-8
OCTANTS, NODES, ITERATIONS = 5.6, 0.68, 7


def work(case):
    """Bytes: points in, 16-byte records out; an operator reads each element's 8 node ids and its
    type once (36 bytes), x once, and writes y once; a mesh is built from 16-byte records.  A solve
    makes four operator applications per V-cycle and level (levels shrink about 2.7-fold), one more
    per CG iteration.  An application is 64 multiply-adds per element."""
    if case["kind"] == "batch":
        n = case["clouds"] * (case["hi"] - case["lo"]) / max(1e-9, np.log(case["hi"] / case["lo"]))
    else:
        n = case["n"]
    e = OCTANTS * n
    v = NODES * e
    build = {"bytes": 24 * n + 16 * e, "flops": 0}

    def applied(size, times):
        return {"bytes": times * (36 * e + 2 * size * v), "flops": times * 128 * e}

    def both(a, b):
        return {k: a[k] + b[k] for k in a}

    if case["kind"] in ("build", "batch"):
        return build
    if case["kind"] == "mesh":
        return both({"bytes": 16 * e, "flops": 0}, applied(8, 1))
    if case["kind"] == "apply":
        return applied(case["precision"] // 8, 1)
    size = case.get("precision", 32) // 8
    solve = both(applied(size, 4 * ITERATIONS * 1.6), applied(8, ITERATIONS))
    return solve if case["kind"] == "solve" else both(build, solve)


# ---- the same in 64 bits with plain torch ---------------------------------------------------------
LEVELS = 20  # deep enough for these clouds: coordinates in units of 2^-20, packed in 63 bits


def _pack(c):
    return c[..., 0] | c[..., 1] << 21 | c[..., 2] << 42


def _unpack(p):
    return torch.stack([p & 0x1FFFFF, p >> 21 & 0x1FFFFF, p >> 42], -1)


def _morton(c):
    key = torch.zeros_like(c[:, 0])
    for bit in range(LEVELS):
        for axis in range(3):
            key |= (c[:, axis] >> bit & 1) << (3 * bit + axis)
    return key


def _member(values, table):
    """(whether, where) of each value in a sorted table."""
    at = torch.searchsorted(table, values).clamp(max=max(0, len(table) - 1))
    return table[at] == values, at


def _leaves(points):
    """The balanced octree, sorted by Morton order: anchors (in units of 2^-LEVELS) and levels."""
    cell = (points * float(1 << DEPTH)).to(torch.int64) >> (DEPTH - LEVELS)
    if len(torch.unique(_pack(cell))) != len(cell):
        return None
    bits = torch.tensor([[k & 1, k >> 1 & 1, k >> 2] for k in range(8)], device=points.device)
    inner = torch.empty(0, dtype=torch.int64, device=points.device)  # subdivided octants of the level below
    anchors, levels = [], []
    for level in range(LEVELS - 1, -1, -1):
        own, count = torch.unique(_pack(cell >> (LEVELS - level)), return_counts=True)
        own = own[count > 1]
        if len(inner):  # an octant is subdivided where a subdivided one touches it from below
            q = _unpack(inner)
            out = 2 * (q & 1) - 1
            near = ((q >> 1).unsqueeze(1) + out.unsqueeze(1) * bits).reshape(-1, 3)
            near = near[((near >= 0) & (near < 1 << level)).all(1)]
            own = torch.unique(torch.cat([own, _pack(near)]))
        if len(own):
            child = (2 * _unpack(own).unsqueeze(1) + bits).reshape(-1, 3)
            if len(inner):
                child = child[~_member(_pack(child), inner)[0]]
            anchors.append(child << (LEVELS - level - 1))
            levels.append(torch.full((len(child),), level + 1, device=points.device))
        inner = own
    anchors, levels = torch.cat(anchors), torch.cat(levels)
    order = torch.argsort(_morton(anchors))
    return anchors[order], levels[order]


def _matrices(device):
    """Trilinear stiffness and mass on [-1, 1]^3."""
    a = np.array([[0.5, -0.5], [-0.5, 0.5]])
    m = np.array([[2.0, 1.0], [1.0, 2.0]]) / 3.0

    def kron(z, y, x):
        return np.kron(z, np.kron(y, x))

    k = kron(m, m, a) + kron(m, a, m) + kron(a, m, m)
    return (torch.tensor(t, device=device) for t in (k, kron(m, m, m)))


class _Mesh:
    """Elements with vertices numbered from the child's own corner of its parent (r = k ^ child), so that
    one of two dozen hanging patterns names an element's interpolation and its matrices."""

    def __init__(self, anchors, levels):
        dev = anchors.device
        size, top = (1 << (LEVELS - levels)).unsqueeze(1), 1 << LEVELS
        child = (anchors // size) & 1
        parent = anchors - child * size
        table, where = torch.sort(_pack(anchors))
        out = (2 * child - 1) * 2 * size
        bits = torch.tensor([[k & 1, k >> 1 & 1, k >> 2] for k in range(8)], device=dev)
        coarse = []
        for s in range(8):  # the parent's neighbour across face or edge s is a leaf of its size
            at = parent + out * bits[s]
            found, j = _member(_pack(at.clamp(0, top - 1)), table)
            inside = ((at >= 0) & (at < top)).all(1) & (levels > 1)
            coarse.append(found & inside & (levels[where[j]] == levels - 1))
        hang = torch.zeros((len(anchors), 8), dtype=torch.bool, device=dev)  # by relative vertex
        for r in range(1, 7):
            for s in range(1, 7):
                if s & (7 & ~r) == s:
                    hang[:, r] |= coarse[s]
        corner = child[:, 0] | child[:, 1] << 1 | child[:, 2] << 2
        vertex = torch.arange(8, device=dev)
        at_top = ((anchors + size) == top).to(torch.int64)
        top_bits = (at_top[:, 0] | at_top[:, 1] << 1 | at_top[:, 2] << 2).unsqueeze(1)
        # nodes in element order: the anchor, and the vertices on the far faces of the domain
        owned = ((vertex & top_bits) == vertex) & ~torch.gather(hang, 1, vertex ^ corner.unsqueeze(1))
        e, k = torch.nonzero(owned, as_tuple=True)
        self.node = anchors[e] + bits[k] * size[e]
        table, where = torch.sort(_pack(self.node))
        self.edge = ((self.node == 0) | (self.node == top)).any(1)
        pattern = (hang.to(torch.int64) << vertex).sum(1)
        order = torch.argsort(pattern)
        self.h = 2.0 ** -levels[order].to(torch.float64).unsqueeze(1)
        kinds, count = torch.unique(pattern, return_counts=True)
        self.slices = []
        stiff, mass = _matrices(dev)
        start = 0
        for p, n in zip(kinds.tolist(), count.tolist()):
            w = torch.zeros((8, 8), dtype=torch.float64, device=dev)
            for r in range(8):
                from_ = [s for s in range(8) if s & r == s] if p >> r & 1 else [r]
                w[r, from_] = 1.0 / len(from_)
            self.slices.append((slice(start, start + n), w.T @ stiff @ w, w.T @ mass @ w))
            start += n
        self.conn = torch.empty((len(anchors), 8), dtype=torch.int64, device=dev)
        for r in range(8):
            k = bits[corner ^ r]
            v = torch.where(hang[:, r : r + 1], parent + 2 * size * k, anchors + size * k)
            found, j = _member(_pack(v), table)
            assert bool(found.all())
            self.conn[:, r] = where[j][order]

    def apply(self, x, lap=1.0, mass=1.0):
        xe = x[self.conn]
        ye = torch.empty_like(xe)
        for part, k, m in self.slices:
            h = self.h[part]
            ye[part] = (xe[part] @ k) * (0.5 * lap * h) + (xe[part] @ m) * (0.125 * mass * h**3)
        return torch.zeros_like(x).index_add_(0, self.conn.reshape(-1), ye.reshape(-1))

    def diagonal(self):
        ye = torch.empty(self.conn.shape, dtype=torch.float64, device=self.conn.device)
        for part, k, m in self.slices:
            h = self.h[part]
            ye[part] = 0.5 * h * torch.diagonal(k) + 0.125 * h**3 * torch.diagonal(m)
        return torch.zeros(len(self.node), dtype=torch.float64, device=ye.device).index_add_(
            0, self.conn.reshape(-1), ye.reshape(-1))

    def poisson(self):
        """-lap u + u = f with u = 0 on the boundary, by CG with the diagonal."""
        free = (~self.edge).to(torch.float64)
        b = self.apply(_load(self.node.to(torch.float64) / float(1 << LEVELS)), lap=0.0) * free
        inv = free / self.diagonal()
        x, r = torch.zeros_like(b), b.clone()
        p = z = inv * r
        rz = r @ z
        bound = 1e-12 * float(torch.linalg.vector_norm(b))
        for it in range(20000):
            q = self.apply(p) * free
            alpha = rz / (p @ q)
            x, r = x + alpha * p, r - alpha * q
            if it % 20 == 19 and float(torch.linalg.vector_norm(r)) < bound:
                break
            z = inv * r
            rz, last = r @ z, rz
            p = z + (rz / last) * p
        return x


def exact(case, seed):
    kind = case["kind"]
    if kind in ("build", "batch"):
        return None  # integer records
    if kind in ("request", "solve") and case["n"] > 600000:
        return None  # CG without multigrid takes too long
    gen = _generator(seed)
    leaves = _leaves(_points(case["cloud"], case["n"], gen))
    if leaves is None:
        return None
    mesh = _Mesh(*leaves)
    if kind in ("request", "solve"):
        y = mesh.poisson()
    else:
        y = mesh.apply(_vector(len(mesh.node), case.get("precision", 64), gen).to(torch.float64))
    out = _room(case["n"], ROOM_NODES)
    _head(out, len(y)).copy_(y)
    return out
