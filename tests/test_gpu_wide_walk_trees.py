"""Closest hits of the wide traversal kernels in trees made by hand, where the
reference walk meets a triangle before a nearer box hides it. The ray is the
same for every path (an orthographic camera of no extent), so that a tree
decides the order of the walk. Accumulators equal the oracle's bit for bit.

The tree, by distance along the ray (boxes in brackets):

    root  L  D [0.4, 0.6], met first, its triangle off the ray
             X [1.8, ...]: X1 (the triangle S, an idle one), an idle one
          R  [1.5, 1.7]: H at 1.6, idle ones

The reference walks L first, so S is taken wherever it is hit. The wide walk
meets R before X, and must not let H, at 1.6, hide S at less than that."""
from __future__ import annotations

import ctypes as C
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32
O = np.asarray([0.3, 0.2, 3.0], F)
D = (np.asarray([0.4, 0.1, -1.0]) / np.linalg.norm([0.4, 0.1, -1.0])).astype(F)
W, H = 31, 23


def _at(t):
    return O.astype(float) + D.astype(float) * t


def _hits(tri):
    """The watertight test of the rays' common ray against (n, 3, 3) triangles
    in single precision: the distances, NaN where it misses."""
    a, b, c = (tri[:, k] - O for k in range(3))
    sx, sy, sz = D[0] / D[2], D[1] / D[2], F(1) / D[2]   # the dominant axis is z; d.z < 0 swaps x and y
    (ax, ay), (bx, by), (cx, cy) = ((v[:, 1] - sy * v[:, 2], v[:, 0] - sx * v[:, 2]) for v in (a, b, c))
    u, v, w = cx * by - cy * bx, ax * cy - ay * cx, bx * ay - by * ax
    mixed = ((u < 0) | (v < 0) | (w < 0)) & ((u > 0) | (v > 0) | (w > 0))
    det = u + v + w
    with np.errstate(divide="ignore", invalid="ignore"):
        t = (u * (sz * a[:, 2]) + v * (sz * b[:, 2]) + w * (sz * c[:, 2])) * (F(1) / det)
    return np.where(mixed | (det == 0), F(np.nan), t)


def _sliver():
    """A triangle in a plane with the ray, which it crosses at 2, from 1 to 3
    along it: a hit is at any of these distances, as the rounding falls. One
    that is hit before its box begins sideways (at 1.8) and before 1.5."""
    r = np.random.default_rng(5)
    n = 400000
    t = np.stack([np.full(n, 1.0), np.full(n, 3.0), r.uniform(1.2, 2.8, n)], 1)
    k = np.stack([np.full(n, 1.0), np.full(n, -1.0), r.uniform(-0.9, 0.9, n)], 1)
    side = np.stack([r.uniform(0.44, 0.46, n), r.uniform(0.04, 0.06, n), np.zeros(n)], 1)
    tri = (_at(0) + D.astype(float) * t[..., None] + k[..., None] * side[:, None, :]).astype(F)
    hit = _hits(tri)
    with np.errstate(divide="ignore"):
        enter = ((tri.min(1) - O) / D)[:, :2].max(1)
    ok = (hit > 1.05) & (hit < 1.45) & (enter > 1.75)
    assert ok.any()
    return tri[ok][0]


def _facing(t, size=0.02):
    c = _at(t)
    return np.asarray([c + (-size, -size, 0), c + (size, -size, 0), c + (0, size, 0)], F)


def _idle(lo, hi):
    """A small triangle in the corner of a box, off the ray."""
    lo, hi = np.asarray(lo, float), np.asarray(hi, float)
    e = (hi - lo) * 0.02
    return np.asarray([lo, lo + (e[0], 0, e[2]), lo + (0, e[1], e[2])], F)


def _box(t0, t1, r):
    p, q = _at(t0), _at(t1)
    return np.minimum(p, q) - (r, r, 0), np.maximum(p, q) + (r, r, 0)


def _tree(s_tri, s_box):
    """Binary nodes as (lo, hi, children or triangle)."""
    near = _box(0.4, 0.6, 0.3)
    r_box = _box(1.5, 1.7, 0.1)

    def idle(b):
        return (*b, _idle(*b))

    def over(*kids):
        return (np.min([k[0] for k in kids], 0), np.max([k[1] for k in kids], 0), list(kids))
    chain = over(idle(r_box), idle(r_box))
    for _ in range(9):
        chain = over(idle(r_box), chain)
    right = over((*_box(1.59, 1.61, 0.05), _facing(1.6)), chain)
    x1 = over((*s_box, s_tri), idle(s_box))
    x = over(x1, idle(s_box))
    return over(over(idle(near), x), right)


def _flatten(root):
    words, tris, level = [None], [], [(root, 0)]
    while level:
        after = []
        for (lo, hi, what), at in level:
            if isinstance(what, list):
                first, count = len(words), 0
                words += [None, None]
                after += [(kid, first + k) for k, kid in enumerate(what)]
            else:
                first, count = len(tris), 1
                tris.append(what)
            w = np.zeros(8, np.uint32)
            w[:3], w[4:7] = np.asarray(lo, F).view(np.uint32), np.asarray(hi, F).view(np.uint32)
            w[3], w[7] = first, count
            words[at] = w
        level = after
    return np.concatenate(words), tris


def _prepared(pkg, s_tri, s_box):
    """The scene of the tree's triangles, the tree in place of its own."""
    nodes, tris = _flatten(_tree(s_tri, s_box))
    key = s_tri.tobytes()
    s = pkg.Scene()
    mats = [s.add_material(pkg.material(base_color=(*c, 1.0), double_sided=1, unlit=1)) for c in
            ((0.9, 0.1, 0.1), (0.1, 0.9, 0.1))]
    for t in tris:
        s.add_mesh(t[None], mats[t.tobytes() == key])
    s.add_light(0, direction=(0.0, -1.0, 0.0), intensity=1.0)
    s.add_camera(tuple(_at(0)), tuple(_at(2)), 0.9, orthographic=True, ymag=1.0)
    p = pkg.prepare(s, pkg.RenderOptions(width=W, height=H, scene_camera=0,
                                         path_trace=pkg.PathTraceOptions(samples_per_pixel=2, max_bounces=3)))
    old = p.geom[8 * p.node_count:].reshape(-1, 12)
    pos = old.view(F)[:, [0, 1, 2, 4, 5, 6, 8, 9, 10]]
    order = [int(np.flatnonzero((pos == t.reshape(-1)).all(1))[0]) for t in tris]
    attrs = p.attrs.reshape(-1, 48)[order].reshape(-1).copy()
    params = type(p.params).from_buffer_copy(bytes(p.params))
    params.env[3], params.offs2[2] = len(nodes) // 8, len(nodes) // 4
    for k in range(3):
        params.eye[k], params.forward[k], params.side[k], params.up[k] = O[k], D[k], 0.0, 0.0
    return dataclasses.replace(p, geom=np.concatenate([nodes, old[order].reshape(-1)]), attrs=attrs,
                               node_count=len(nodes) // 8, params=params)


class _Ctx:
    def __init__(self, N):
        self.N, self.L = N, N.lib()
        self.h = C.c_void_p()
        assert self.L.oxpt_create(0, C.byref(self.h)) == 0
        self.ok(self.L.oxpt_resize(self.h, W, H))

    def ok(self, st):
        assert st == 0, self.L.oxpt_last_error(self.h).decode()

    def load(self, p, staged):
        d = self.N.SceneDesc(p.geom.ctypes.data, p.geom.size, p.attrs.ctypes.data, p.attrs.size, p.atlas.ctypes.data,
                             p.atlas_side, p.atlas_layers, p.node_count, p.slot_count)
        if staged:
            self.ok(self.L.oxpt_stage_scene(self.h, C.byref(d), p.tables.ctypes.data, p.tables.size))
        else:
            self.ok(self.L.oxpt_upload_scene(self.h, C.byref(d)))
            self.ok(self.L.oxpt_set_tables(self.h, p.tables.ctypes.data, p.tables.size))
        params = p.params
        self.ok(self.L.oxpt_set_params(self.h, C.byref(params)))
        self.ok(self.L.oxpt_reset(self.h))

    def accum(self):
        out = np.empty((H, W, 4), F)
        self.ok(self.L.oxpt_read_accum(self.h, out.ctypes.data))
        self.ok(self.L.oxpt_finish(self.h))
        return out


def _same(pkg, oracle, p, staged):
    cpu, _ = oracle.render(p, 2)
    assert (cpu[..., 1] > 0.5).all() and (cpu[..., 0] < 0.5).all()  # S, not H, in every pixel
    c, ex = _Ctx(pkg._native), _Ctx(pkg._native)
    try:
        c.load(p, staged)
        c.ok(c.L.oxpt_refine(c.h, 0, 2))
        four = (C.c_uint32 * 4)()
        c.ok(c.L.oxpt_diag_bvh4(c.h, four))
        assert four[0]  # the tree has its four-wide form
        assert np.array_equal(c.accum().view(np.uint32), cpu.view(np.uint32))
        if staged:  # (such a context is traced by its own refine alone)
            return
        c.ok(c.L.oxpt_reset(c.h))
        frame = (pkg._native.BatchFrame * 1)(pkg._native.BatchFrame(c.h, 0, 2, 0, H))
        ex.ok(ex.L.oxpt_refine_batch(ex.h, frame, 1))
        assert np.array_equal(c.accum().view(np.uint32), cpu.view(np.uint32))
    finally:
        c.L.oxpt_destroy(c.h)
        c.L.oxpt_destroy(ex.h)


@pytest.mark.parametrize("staged", [False, True])
def test_sliver_hit_before_its_box_begins(pkg, oracle, staged):
    s = _sliver()
    _same(pkg, oracle, _prepared(pkg, s, (s.min(0), s.max(0))), staged)


@pytest.mark.parametrize("staged", [False, True])
@pytest.mark.parametrize("hit", [1.0, 1.45])
def test_triangle_outside_its_leafs_box(pkg, oracle, hit, staged):
    _same(pkg, oracle, _prepared(pkg, _facing(hit), _box(1.8, 2.4, 0.05)), staged)
