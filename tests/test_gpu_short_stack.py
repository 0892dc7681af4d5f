"""The short-stack traversal kernels (csrc/wave_walk.cu) where they still run
in an ordinary refine: scenes whose four-wide tree is refused (closest hits
and shadow rays walk the binary tree) and scenes whose leaves do not hold
their triangles (closest hits alone). Accumulators equal the oracle's bit for
bit, whatever part of the stack and of the tree is kept on chip."""
from __future__ import annotations

import ctypes as C
import dataclasses

import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

W, H, SPP = 48, 32, 3


def _prepared(pkg, which):
    """A prepared scene with one leaf's box made larger than its parent's
    ("refused") or smaller than its triangles ("outside")."""
    scene = pkg.Scene.icosphere(freq=24, seed=5, n_materials=8, n_textures=2, tex_size=64, n_punctual=4, n_emissive=32,
                                material_mix=1) if which[0] == "layered" else scenes.alpha_scene(pkg)
    p = pkg.prepare(scene, pkg.RenderOptions(width=W, height=H, scene_camera=0, path_trace=pkg.PathTraceOptions(
        samples_per_pixel=SPP, max_bounces=6)), pkg.EnvironmentMap.sky(64, 32) if which[0] == "layered" else None)
    geom = p.geom.copy()
    nodes = geom[:8 * p.node_count].reshape(-1, 8)
    leaf = int(np.flatnonzero(nodes[:, 7])[-1])
    box = nodes[leaf].view(np.float32)
    if which[1] == "refused":
        box[4:7] = nodes[0].view(np.float32)[4:7] + 1.0
    else:
        box[4:7] = 0.5 * (box[:3] + box[4:7])
    return dataclasses.replace(p, geom=geom)


class _Ctx:
    def __init__(self, pkg, p=None, **tuning):
        self.N, self.L = pkg._native, pkg._native.lib()
        self.h = C.c_void_p()
        assert self.L.oxpt_create(0, C.byref(self.h)) == 0
        t = self.N.Tuning()
        self.ok(self.L.oxpt_get_tuning(self.h, C.byref(t)))
        for k, v in tuning.items():
            setattr(t, k, v)
        self.ok(self.L.oxpt_set_tuning(self.h, C.byref(t)))
        if p is None:
            return
        self.ok(self.L.oxpt_resize(self.h, W, H))
        d = self.N.SceneDesc(p.geom.ctypes.data, p.geom.size, p.attrs.ctypes.data, p.attrs.size, p.atlas.ctypes.data,
                             p.atlas_side, p.atlas_layers, p.node_count, p.slot_count)
        self.ok(self.L.oxpt_upload_scene(self.h, C.byref(d)))
        self.ok(self.L.oxpt_set_tables(self.h, p.tables.ctypes.data, p.tables.size))
        params = p.params
        self.ok(self.L.oxpt_set_params(self.h, C.byref(params)))
        self.ok(self.L.oxpt_reset(self.h))

    def ok(self, st):
        assert st == 0, self.L.oxpt_last_error(self.h).decode()

    def four_wide(self):
        four = (C.c_uint32 * 4)()
        self.ok(self.L.oxpt_diag_bvh4(self.h, four))
        return bool(four[0])

    def refine(self):
        self.ok(self.L.oxpt_refine(self.h, 0, SPP))
        return self.accum()

    def accum(self):
        out = np.empty((H, W, 4), np.float32)
        self.ok(self.L.oxpt_read_accum(self.h, out.ctypes.data))
        self.ok(self.L.oxpt_finish(self.h))
        return out

    def __del__(self):
        self.L.oxpt_destroy(self.h)


SCENES = [("layered", "refused"), ("alpha", "refused"), ("layered", "outside")]


@pytest.mark.parametrize("window", [0, 1])
@pytest.mark.parametrize("lim,stage", [(0, 0), (1, 200), (3, 0), (16, 511)])
@pytest.mark.parametrize("mode,variant", [(1, 3), (2, 4), (2, 5)])
@pytest.mark.parametrize("which", SCENES)
def test_on_chip_parts_bit_exact(pkg, oracle, which, mode, variant, lim, stage, window):
    p = _prepared(pkg, which)
    c = _Ctx(pkg, p, mode=mode, trace_variant=variant, wave_slots=500)
    assert c.four_wide() == (which[1] == "outside")
    c.ok(c.L.oxpt_diag_set_walk(c.h, lim, stage))
    c.ok(c.L.oxpt_diag_set_l2_window(c.h, window, None))
    got = c.refine()
    c.ok(c.L.oxpt_diag_set_l2_window(c.h, 0, None))
    want, _ = oracle.render(p, SPP)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("graphs", [0, 1])
def test_mixed_batch_bit_exact(pkg, oracle, graphs):
    """A scene with the wide walk beside others without it."""
    ps = [_prepared(pkg, w) for w in SCENES]
    ps.append(pkg.prepare(scenes.materials_scene(pkg), pkg.RenderOptions(width=W, height=H)))
    for group in (ps, ps[2:], ps[3:]):
        cs = [_Ctx(pkg, p) for p in group]
        ex = _Ctx(pkg, mode=2, trace_variant=4, graphs=graphs, wave_slots=900)
        frames = (pkg._native.BatchFrame * len(cs))(*(pkg._native.BatchFrame(c.h, 0, SPP, 0, H) for c in cs))
        ex.ok(ex.L.oxpt_refine_batch(ex.h, frames, len(cs)))
        for p, c in zip(group, cs):
            want, _ = oracle.render(p, SPP)
            assert np.array_equal(c.accum().view(np.uint32), want.view(np.uint32))
