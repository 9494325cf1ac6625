"""Tagging by tiles (voxel.cu): the images that a tile of corners leaves out are
those that no corner of it is in. Against the primitives' own tests in numpy,
every operation and periodic image at every corner, bit for bit: flips, periodic
axes, grids thinner than a tile, one corner, corners on surfaces, primitives
that reach in through the periodic boundary and primitives that cover tiles."""
import ctypes as C

import numpy as np
import pytest

from aether_b200 import _abi as A

_P = C.POINTER


def op(kind, mat, *p):
    o = A.StructureOp()
    o.kind, o.mat_index = kind, mat
    for i, v in enumerate(p):
        o.p[i] = v
    return o


def inside(o, x, y, z):
    p = [o.p[t] for t in range(16)]
    if o.kind == A.OP_BLOCK:
        b = [sorted(p[2 * t:2 * t + 2]) for t in range(3)]
        return ((x >= b[0][0]) & (x < b[0][1]) & (y >= b[1][0]) & (y < b[1][1]) & (z >= b[2][0]) & (z < b[2][1]))
    if o.kind == A.OP_LAYER:
        v = (x, y, z)[int(p[0])]
        return (v >= p[1]) & (v < p[2]) & (x == x) & (y == y) & (z == z)
    if o.kind == A.OP_SPHERE:
        ex, ey, ez = x - p[0], y - p[1], z - p[2]
        return ex * ex + ey * ey + ez * ez <= p[3] * p[3]
    if o.kind == A.OP_ELLIPSOID:
        box = ~((x < p[0] - p[3]) | (x > p[0] + p[3]) | (y < p[1] - p[4]) | (y > p[1] + p[4]) | (z < p[2] - p[5]) |
                (z > p[2] + p[5]))
        ex, ey, ez = (x - p[0]) / p[3], (y - p[1]) / p[4], (z - p[2]) / p[5]
        return box & (ex * ex + ey * ey + ez * ez <= 1.0)
    # cylinder and cone
    r = p[6]
    v = [p[3] - p[0], p[4] - p[1], p[5] - p[2]]
    length = np.sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2])
    b = [t / length for t in v]
    box = ~((x < min(p[0], p[3]) - r) | (x > max(p[0], p[3]) + r) | (y < min(p[1], p[4]) - r) |
            (y > max(p[1], p[4]) + r) | (z < min(p[2], p[5]) - r) | (z > max(p[2], p[5]) + r))
    ex, ey, ez = x - p[0], y - p[1], z - p[2]
    proj = b[0] * ex + b[1] * ey + b[2] * ez
    ex, ey, ez = ex - proj * b[0], ey - proj * b[1], ez - proj * b[2]
    rt = ex * ex + ey * ey + ez * ez
    r2 = r * r
    if o.kind == A.OP_CONE:
        r2 = r * (1.0 - proj / length)
        r2 = r2 * r2
    return box & (proj >= 0) & (proj <= length) & (rt <= r2)


def numpy_tags(n, d, ops, default, periodic, flip, lengths):
    axes = []
    for t in range(3):
        v = np.arange(n[t]) * d[t]
        if flip[t]:
            v = lengths[t] - v
        if periodic[t]:
            while (v < 0).any():
                v = np.where(v < 0, v + lengths[t], v)
            while (v >= lengths[t]).any():
                v = np.where(v >= lengths[t], v - lengths[t], v)
        axes.append(v)
    z, y, x = np.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    out = np.full(x.shape, default, np.uint32)
    for o in ops:
        hit = np.zeros(x.shape, bool)
        for ii in range(-periodic[0], periodic[0] + 1):
            for jj in range(-periodic[1], periodic[1] + 1):
                for kk in range(-periodic[2], periodic[2] + 1):
                    hit |= inside(o, x + ii * lengths[0], y + jj * lengths[1], z + kk * lengths[2])
        out[hit] = o.mat_index
    return out


def device_tags(n, d, ops, default, periodic, flip, lengths):
    from aether_b200 import _lib
    out = np.zeros(n[0] * n[1] * n[2], np.uint32)
    arr = (A.StructureOp * max(len(ops), 1))(*ops)
    desc = A.structure_desc(default, periodic, flip, lengths)
    _lib.check(_lib.load().aefdtd_discretize(None, n[0], n[1], n[2], d[0], d[1], d[2], arr, len(ops), C.byref(desc),
                                             out.ctypes.data_as(_P(C.c_uint32)), 0))
    return out.reshape(n[2], n[1], n[0])


def scene(rng, d, lengths, count):
    def at(t):   # some coordinates on corners
        v = rng.uniform(-0.1, 1.1) * lengths[t]
        return round(v / d[t]) * d[t] if rng.random() < 0.5 else v
    ops = [op(A.OP_LAYER, 1, 2.0, 0.0, 0.4 * lengths[2])]
    size = min(max(v, 40e-9) for v in lengths)
    for _ in range(count):
        m = int(rng.integers(1, 9))
        k = int(rng.choice([A.OP_BLOCK, A.OP_LAYER, A.OP_SPHERE, A.OP_SPHERE, A.OP_CYLINDER, A.OP_CONE, A.OP_ELLIPSOID]))
        c = [at(t) for t in range(3)]
        if k == A.OP_BLOCK:
            e = [at(t) for t in range(3)]
            ops.append(op(k, m, c[0], e[0], c[1], e[1], c[2], e[2]))
        elif k == A.OP_LAYER:
            ops.append(op(k, m, float(rng.integers(0, 3)), c[2], c[2] + rng.uniform(0, 0.1) * size))
        elif k == A.OP_SPHERE:
            ops.append(op(k, m, *c, rng.integers(1, 8) * d[0] if rng.random() < 0.5 else rng.uniform(0.02, 0.2) * size))
        elif k == A.OP_ELLIPSOID:
            ops.append(op(k, m, *c, *(rng.uniform(0.05, 0.3, 3) * size)))
        else:
            ops.append(op(k, m, *c, *[v + rng.uniform(-0.3, 0.3) * size for v in c], rng.uniform(0.05, 0.2) * size))
    return ops


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(37, 29, 45), (1, 1, 1), (1, 1, 300), (300, 2, 3), (5, 200, 1), (64, 33, 17), (33, 4, 9)])
@pytest.mark.parametrize("periodic,flip", [((0, 0, 0), (0, 0, 0)), ((1, 1, 0), (1, 0, 1)), ((1, 1, 1), (0, 1, 0))])
def test_tags_equal_every_test_at_every_corner(n, periodic, flip):
    rng = np.random.default_rng(n[0] + 7 * n[2] + sum(periodic))
    d = (2.5e-9, 3e-9, 2e-9)
    lengths = tuple(n[t] * d[t] for t in range(3))
    for count in (0, 6, 40):
        ops = scene(rng, d, lengths, count)
        want = numpy_tags(n, d, ops, 9, periodic, flip, lengths)
        assert np.array_equal(device_tags(n, d, ops, 9, periodic, flip, lengths), want)


@pytest.mark.gpu
def test_an_image_that_covers_every_tile_ends_the_list():
    n, d = (70, 40, 30), (1e-9,) * 3
    lengths = (70e-9, 40e-9, 30e-9)
    ops = scene(np.random.default_rng(1), d, lengths, 20) + [op(A.OP_BLOCK, 5, -1, 1, -1, 1, -1, 1)]
    ops += [op(A.OP_SPHERE, 6, 20e-9, 20e-9, 15e-9, 9e-9)]
    got = device_tags(n, d, ops, 0, (1, 1, 0), (0, 0, 0), lengths)
    assert np.array_equal(got, numpy_tags(n, d, ops, 0, (1, 1, 0), (0, 0, 0), lengths))
    assert set(np.unique(got)) == {5, 6}
