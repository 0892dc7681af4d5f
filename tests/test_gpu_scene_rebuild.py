"""One tracer synced to scenes of very different sizes in turn: builds reuse
its scene buffers and scratch block, and each scene's buffers and frame are
those of a tracer that never held another (equal word for word)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(pkg, n, seed, copies=1):
    """n random triangles; with `copies`, each repeated (equal boxes and costs)."""
    r = np.random.default_rng(seed)
    p = (r.uniform(-1, 1, (n, 1, 3)) + r.uniform(-0.2, 0.2, (n, 3, 3))).astype(np.float32)
    s = pkg.Scene()
    m = s.add_material(pkg.material(base_color=(0.7, 0.6, 0.5, 1.0), double_sided=1))
    s.add_mesh(np.concatenate([p] * copies), m)
    s.add_camera((1.5, 1.2, 3.0), (0.0, 0.0, 0.0), 0.9)
    s.add_light(1, position=(1.0, 2.0, 1.0), intensity=6.0)
    return s


def _scenes(pkg):
    yield _soup(pkg, 40, 1)
    yield pkg.Scene.icosphere(freq=40, seed=3, n_materials=4, n_textures=2, tex_size=64, n_punctual=2, n_emissive=9,
                              material_mix=1)
    for n, copies in ((1, 1), (2, 1), (7, 1), (8, 1), (9, 1), (3, 3), (1, 20), (33, 1), (1024, 1), (1025, 1)):
        yield _soup(pkg, n, n, copies)
    yield pkg.Scene.icosphere(freq=41, seed=4, n_materials=4, n_textures=1, tex_size=128, n_punctual=1, n_emissive=3,
                              material_mix=1)
    yield pkg.Scene.box_field(700, seed=2)


def test_rebuilt_scenes_equal_fresh_ones(pkg):
    opts = pkg.RenderOptions(width=30, height=20, path_trace=pkg.PathTraceOptions(samples_per_pixel=2, max_bounces=4))
    kept = pkg.GpuPathTracer(0)
    for scene in _scenes(pkg):
        frames = []
        for t in (kept, pkg.GpuPathTracer(0)):
            t.invalidate_scene()
            assert t.sync(scene, opts)
            t.refine(2)
            t.finish()
            frames.append((t.read_accum(), t.prepared()))
        host = pkg.prepare(scene, opts)
        for acc, p in frames:
            assert np.array_equal(acc.view(np.uint32), frames[1][0].view(np.uint32))
            for name in ("geom", "attrs", "tables", "atlas"):
                a, b = getattr(p, name), getattr(host, name)
                assert a.shape == b.shape and np.array_equal(a.view(np.uint8), b.view(np.uint8)), name
