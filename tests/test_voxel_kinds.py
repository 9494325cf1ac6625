"""The voxeliser's other kinds (sine layers, vector blocks and triangles,
meshes, coatings) beside the plain ones, against their tests in numpy at every
corner, every operation and every periodic image: what tagging by tiles leaves
out contains no corner. Vector blocks, triangles and meshes are compared where a
corner is not within 1e-9 (relative) of a face, as their solves round."""
import math

import numpy as np
import pytest

from aether_b200 import _abi as A
from test_voxel import icosphere
from test_voxel_tiles import device_tags, inside, op, scene

pytestmark = pytest.mark.gpu
NEAR = 1e-9


class Tags:
    """Structure::index in numpy. unsure: corners too near to a face to say."""

    def __init__(self, ops, default, periodic, flip, lengths, meshes=()):
        self.ops, self.default, self.periodic, self.flip, self.lengths = ops, default, periodic, flip, lengths
        self.meshes = meshes
        self.seeds = {}

    def fold(self, v, axis):
        L = self.lengths[axis]
        v = L - v if self.flip[axis] else v
        if self.periodic[axis]:
            while (v < 0).any():
                v = np.where(v < 0, v + L, v)
            while (v >= L).any():
                v = np.where(v >= L, v - L, v)
        return v

    def index(self, x, y, z, level=None):
        """Tags and the unsure mask of points (flat arrays)."""
        level = len(self.ops) if level is None else level
        x, y, z = self.fold(x, 0), self.fold(y, 1), self.fold(z, 2)
        out = np.full(x.shape, -1, np.int64)
        unsure = np.zeros(x.shape, bool)
        p, L = self.periodic, self.lengths
        for q in range(level - 1, -1, -1):
            for ii in range(-p[0], p[0] + 1):
                for jj in range(-p[1], p[1] + 1):
                    for kk in range(-p[2], p[2] + 1):
                        at = np.nonzero(out == -1)[0]
                        hit, near = self.hit(q, x[at] + ii * L[0], y[at] + jj * L[1], z[at] + kk * L[2])
                        unsure[at] |= near
                        out[at[hit]] = self.ops[q].mat_index
        out[out == -1] = self.default
        return out, unsure

    def hit(self, q, x, y, z):
        o = self.ops[q]
        p = [o.p[t] for t in range(16)]
        sure = np.zeros(x.shape, bool)
        if len(x) == 0:
            return sure, sure
        if o.kind == A.OP_SIN_LAYER:
            def wave(v, period, phase):
                inv = 0.0 if period == 0 else 1.0 / period
                known = {u: math.sin(2.0 * math.pi * (u * inv + phase)) for u in set(v.tolist())}
                return np.array([known[u] for u in v.tolist()])
            t = 0.5 * (wave(x, p[4], p[5]) + wave(y, p[6], p[7]))
            return (p[0] + p[1] * t <= z) & (p[2] + p[3] * t >= z), sure
        if o.kind in (A.OP_VECT_BLOCK, A.OP_VECT_TRI):
            m = np.array(p[3:12]).reshape(3, 3).T
            a, b, c = np.linalg.solve(m, np.stack([x - p[0], y - p[1], z - p[2]]))
            if o.kind == A.OP_VECT_BLOCK:
                faces = [a, 1 - a, b, 1 - b, c, 1 - c]
            else:
                faces = [b, 1 - b, c, 1 - c, a - c * p[12], 1 - c * (1 - p[12]) - a]
            least = np.min(faces, axis=0)
            return least >= 0, np.abs(least) < NEAR
        if o.kind == A.OP_MESH:
            v, f = self.meshes[int(p[4])]
            v = v * p[3]
            n = np.zeros(x.shape, int)
            near = np.zeros(x.shape, bool)
            d = np.array([0.36, 0.48, 0.8])
            box = (x >= v[:, 0].min()) & (x <= v[:, 0].max()) & (y >= v[:, 1].min()) & (y <= v[:, 1].max()) & \
                  (z >= v[:, 2].min()) & (z <= v[:, 2].max())
            pts = np.stack([x, y, z], 1)
            for t in f:
                e1, e2 = v[t[1]] - v[t[0]], v[t[2]] - v[t[0]]
                s = pts - v[t[0]]
                pv = np.cross(d, e2)
                det = pv @ e1
                qv = np.cross(s, e1)
                u, w, r = (s @ pv) / det, (qv @ d) / det, (qv @ e2) / det
                n += (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & (r >= 0)
                plane = np.abs(s @ np.cross(e1, e2)) / np.linalg.norm(np.cross(e1, e2))
                near |= (plane < NEAR * np.abs(v).max()) | (np.abs(u) < NEAR) | (np.abs(w) < NEAR) | (np.abs(1 - u - w) < NEAR)
            return box & (n % 2 == 1), near & box
        if o.kind == A.OP_COATING:
            return self.coating(q, p, x, y, z)
        if o.kind == A.OP_CONF_COATING:
            return self.conformal(q, p, x, y, z)
        return inside(o, x, y, z), sure

    def coating(self, q, p, x, y, z):
        theta, phi = p[0] * (math.pi / 180.0), p[1] * (math.pi / 180.0)
        d = (math.cos(phi) * math.sin(theta), math.sin(phi) * math.sin(theta), -math.cos(theta))
        t2, delta, origin = p[2] * p[2], p[3], int(p[4])
        tag, unsure = self.index(x, y, z, q)
        ok = tag == origin
        marching, support = ok.copy(), np.zeros(x.shape, bool)
        at = (x, y, z)
        i = 0
        while marching.any():   # along the direction, within the thickness, for something to rest on
            e = [a - b for a, b in zip(at, (x, y, z))]
            marching &= (e[0] * e[0] + e[1] * e[1] + e[2] * e[2] <= t2) & (at[2] > 0)
            s = i * delta
            at = (x + s * d[0], y + s * d[1], z + s * d[2])
            tag, un = self.index(*at, q)
            unsure |= un & marching
            support |= marching & (tag != origin)
            marching &= ~support
            i += 1
        ok &= support
        marching = ok.copy()
        at = (x, y, z)
        i = 0
        while True:   # against it, up to the top: nothing in between
            marching &= at[2] <= self.lengths[2]
            if not marching.any():
                break
            s = i * delta
            at = (x - s * d[0], y - s * d[1], z - s * d[2])
            tag, un = self.index(*at, q)
            unsure |= un & marching
            ok &= ~(marching & (tag != origin))
            marching &= ok
            i += 1
        return ok, unsure

    def conformal(self, q, p, x, y, z):
        thick, delta, origin, L = p[0], p[1] if p[1] > 0 else 5e-9, int(p[2]), self.lengths
        if q not in self.seeds:
            n = [max(0, int(L[t] / delta)) for t in range(3)]
            k, j, i = np.meshgrid(*[np.arange(n[t]) for t in (2, 1, 0)], indexing="ij")
            c = [i.ravel() * delta, j.ravel() * delta, k.ravel() * delta]
            own = self.index(*c, q)[0] == origin
            seeds = []
            for t in range(3):
                for sign in (-1, 1):
                    near = [v + sign * delta if u == t else v for u, v in enumerate(c)]
                    if sign < 0:
                        near[t] = c[t] - delta
                    mark = own & (self.index(*near, q)[0] != origin)
                    seeds.append(np.stack([v[mark] for v in near], 1))
            self.seeds[q] = np.concatenate(seeds)
        tag, unsure = self.index(x, y, z, q)
        ok = tag == origin
        ok &= (x >= 0) & (x <= L[0]) & (y >= 0) & (y <= L[1]) & (z >= 0) & (z <= L[2])
        found = np.zeros(x.shape, bool)
        for s in self.seeds[q]:
            ex, ey, ez = x - s[0], y - s[1], z - s[2]
            found |= ex * ex + ey * ey + ez * ez < thick * thick
        return ok & found, unsure


def corners(n, d):
    z, y, x = np.meshgrid(np.arange(n[2]) * d[2], np.arange(n[1]) * d[1], np.arange(n[0]) * d[0], indexing="ij")
    return x.ravel(), y.ravel(), z.ravel()


def compare(n, d, ops, default, periodic, flip, lengths, meshes=()):
    if meshes:
        got = device_mesh_tags(n, d, ops, default, periodic, flip, lengths, meshes)
    else:
        got = device_tags(n, d, ops, default, periodic, flip, lengths)
    want, unsure = Tags(ops, default, periodic, flip, lengths, meshes).index(*corners(n, d))
    assert unsure.mean() < 0.02
    wrong = (got.ravel() != want) & ~unsure
    assert not wrong.any(), (wrong.sum(), np.argwhere(wrong)[:4].ravel(), got.ravel()[wrong][:4], want[wrong][:4])
    return got


def device_mesh_tags(n, d, ops, default, periodic, flip, lengths, meshes):
    import ctypes as C
    from aether_b200 import _lib
    out = np.zeros(n[0] * n[1] * n[2], np.uint32)
    arr = (A.StructureOp * len(ops))(*ops)
    desc = A.structure_desc(default, periodic, flip, lengths, meshes=list(meshes))
    _lib.check(_lib.load().aefdtd_discretize(None, *n, *d, arr, len(ops), C.byref(desc),
                                             out.ctypes.data_as(C.POINTER(C.c_uint32)), 0))
    return out.reshape(n[2], n[1], n[0])


def more_kinds(rng, lengths, meshes, count):
    """Operations of the kinds that test_voxel_tiles.py leaves out."""
    size, ops = min(lengths), []
    for _ in range(count):
        m = int(rng.integers(1, 9))
        k = int(rng.choice([A.OP_SIN_LAYER, A.OP_VECT_BLOCK, A.OP_VECT_TRI, A.OP_MESH]))
        c = [rng.uniform(-0.1, 0.9) * v for v in lengths]
        if k == A.OP_SIN_LAYER:
            h = rng.uniform(0.1, 0.8) * lengths[2]
            ops.append(op(k, m, h, rng.uniform(0, 0.1) * size, h + 0.1 * size, rng.uniform(0, 0.1) * size,
                          rng.choice([0.0, lengths[0]]), rng.uniform(), lengths[1] / 2, rng.uniform()))
        elif k == A.OP_MESH:
            ops.append(op(k, m, 0.0, 0.0, 0.0, 1.0, float(rng.integers(0, len(meshes)))))
        else:
            v = rng.uniform(-0.35, 0.35, 9) * size
            ops.append(op(k, m, *c, *v, rng.uniform()))
    return ops


@pytest.mark.parametrize("n", [(37, 11, 19), (64, 5, 9), (5, 40, 6), (1, 1, 90)])
@pytest.mark.parametrize("periodic,flip", [((0, 0, 0), (0, 0, 0)), ((1, 1, 0), (1, 0, 1)), ((1, 1, 1), (0, 1, 0))])
def test_every_kind_equals_its_test_at_every_corner(n, periodic, flip):
    rng = np.random.default_rng(3 * n[0] + n[2] + 5 * sum(flip))
    d = (2.5e-9, 3e-9, 2e-9)
    lengths = tuple(n[t] * d[t] for t in range(3))
    meshes = [icosphere([0.31 * v + 0.17e-9 for v in lengths], 0.23 * max(min(lengths), 20e-9), 0),
              icosphere([0.72 * v + 0.13e-9 for v in lengths], 0.31 * max(min(lengths), 20e-9), 0)]
    for count in (2, 7):
        ops = scene(rng, d, lengths, count) + more_kinds(rng, lengths, meshes, count)
        ops = [ops[i] for i in rng.permutation(len(ops))]
        compare(n, d, ops, 9, periodic, flip, lengths, meshes)


@pytest.mark.parametrize("kind,periodic", [(k, p) for k in ("directional", "conformal", "nested", "between")
                                           for p in ((0, 0, 0), (1, 1, 0)) if k != "nested" or p == (0, 0, 0)])
def test_coatings_equal_their_test_at_every_corner(kind, periodic):
    """Coatings are tested at every corner whatever lies around them: above and
    below other operations, with periodic images, over tiles without any."""
    n, d = (40, 10, 18), (2.5e-9,) * 3
    lengths = tuple(v * 2.5e-9 for v in n)
    ops = [op(A.OP_LAYER, 1, 2.0, 0.0, 20e-9), op(A.OP_SPHERE, 1, 30e-9, 14e-9, 20e-9, 10e-9),
           op(A.OP_BLOCK, 2, 5e-9, 16e-9, 13e-9, 24e-9, 15e-9, 32e-9), op(A.OP_CONE, 1, 80e-9, 11e-9, 18e-9, 80e-9, 11e-9, 36e-9, 9e-9)]
    if kind == "directional":
        ops += [op(A.OP_COATING, 3, 20.0, 30.0, 6e-9, 1e-9, 0)]
    elif kind == "conformal":
        ops += [op(A.OP_CONF_COATING, 3, 7.6e-9, 2.5e-9, 0)]
    elif kind == "nested":
        ops += [op(A.OP_CONF_COATING, 3, 5.1e-9, 2.5e-9, 0), op(A.OP_COATING, 4, 0.0, 0.0, 4e-9, 1e-9, 0)]
    else:
        ops += [op(A.OP_COATING, 3, 10.0, 200.0, 5e-9, 1e-9, 0), op(A.OP_SPHERE, 5, 62e-9, 20e-9, 25e-9, 9e-9),
                op(A.OP_ELLIPSOID, 6, 20e-9, 4e-9, 38e-9, 12e-9, 6e-9, 8e-9)]
    got = compare(n, d, ops, 0, periodic, (0, 0, 0), lengths)
    assert (got == 3).sum() > 20
