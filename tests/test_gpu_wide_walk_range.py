"""The wide traversal kernels over the range of coordinates: scenes from a
micrometre to more than the kernels' own range, seen and lit along the axes,
where reciprocal directions are largest. Accumulators equal the oracle's bit
for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(pkg, scale, far, towards, light):
    """A floor and boxes above it, `scale` units to each side of the middle,
    and a triangle out of sight that is `far` units large."""
    c = np.linspace(-1, 1, 7)
    quads = [[(x, 0, z), (x, 0, w), (y, 0, w), (y, 0, z)] for x, y in zip(c, c[1:]) for z, w in zip(c, c[1:])]
    r = np.random.default_rng(3)
    for _ in range(12):
        (x, z), h, b = r.uniform(-0.8, 0.8, 2), r.uniform(0.2, 0.8), 0.12
        for dx, dz in ((-b, -b), (b, -b), (b, b), (-b, b)):
            p, q = (x + dx, z + dz), (x - dz, z + dx)
            quads.append([(p[0], 0, p[1]), (q[0], 0, q[1]), (q[0], h, q[1]), (p[0], h, p[1])])
        quads.append([(x - b, h, z - b), (x - b, h, z + b), (x + b, h, z + b), (x + b, h, z - b)])
    tris = np.asarray([t for q in quads for t in ((q[0], q[1], q[2]), (q[0], q[2], q[3]))])
    s = pkg.Scene()
    s.add_mesh((tris * scale).astype(np.float32),
               s.add_material(pkg.material(base_color=(0.7, 0.6, 0.5, 1.0), double_sided=1)))
    if far:
        s.add_mesh((np.asarray([[(1, 3, 1), (2, 3, 1), (1, 4, 2)]]) * far).astype(np.float32), 0)
    s.add_light(0, direction=light, intensity=3.0)
    d = np.asarray(towards, float)
    s.add_camera(tuple(-2.0 * scale * d), (0.0, 0.0, 0.0), 0.9, up=(0, 0, 1) if d[1] else (0, 1, 0),
                 orthographic=True, ymag=1.1 * scale)
    return s


SCALES = [(1.0e-6, 0), (1.0, 0), (1.0e6, 0), (4.0e6, 0), (1.0e8, 0), (1.0e12, 0), (3.0e17, 0), (3.0e18, 0),
          (1.0, 4.0e6), (1.0, 1.0e12), (1.0, 3.0e17), (1.0, 3.0e18), (1.0, 1.0e30)]
VIEWS = [((0, -1, 0), (0.0, -1.0, 0.0)), ((0, 0, 1), (-0.0, -1.0, -0.0)), ((-1, 0, 0), (1.0, -0.0, 0.0))]


def _tracer(pkg, scale, view, **tuning):
    t = pkg.GpuPathTracer(0)
    t.set_environment(pkg.EnvironmentMap.sky(32, 16))
    t.set_tuning(mode=2, **tuning)
    assert t.sync(_scene(pkg, *scale, *view), pkg.RenderOptions(
        width=31, height=23, path_trace=pkg.PathTraceOptions(samples_per_pixel=2, max_bounces=4)))
    return t


@pytest.mark.parametrize("view", VIEWS)
@pytest.mark.parametrize("scale", SCALES)
def test_axis_rays_at_every_scale(pkg, oracle, scale, view):
    t = _tracer(pkg, scale, view)
    t.refine(2)
    t.finish()
    cpu, _ = oracle.render(t.prepared(), 2)
    assert np.array_equal(t.read_accum().view(np.uint32), cpu.view(np.uint32))
    if scale[0] < 1.0e10:  # (products of three larger edges overflow)
        assert len(np.unique(cpu[..., :3])) > 4  # surfaces and shadows are seen


def test_axis_rays_of_mixed_scales_in_a_batch(pkg, oracle):
    tracers = [_tracer(pkg, s, VIEWS[k % 3]) for k, s in enumerate(SCALES)]
    ex = pkg.GpuPathTracer(0)
    ex.set_tuning(mode=2, graphs=1)
    pkg.refine_batch(tracers, 2, ex)
    for s, t in zip(SCALES, tracers):
        t.finish()
        cpu, _ = oracle.render(t.prepared(), 2)
        assert np.array_equal(t.read_accum().view(np.uint32), cpu.view(np.uint32)), s


def test_small_object_in_a_large_scene_costs_no_more(pkg):
    """A finely tessellated object above a ground of 10 and of 10^5 units: the
    same rays meet the same triangles, so the frames take about as long (a box
    test that widens boxes by a share of the largest coordinate took 450 times
    as long)."""
    import time
    best = []
    for ground in (10.0, 1.0e5):
        s = pkg.Scene.icosphere(freq=160, seed=3, n_materials=2, n_textures=1, tex_size=16, n_punctual=2, n_emissive=0,
                                material_mix=0)
        q = np.asarray([(-1, 0, -1), (-1, 0, 1), (1, 0, 1), (1, 0, -1)], np.float32) * ground - (0, 1.2, 0)
        s.add_mesh(np.asarray([q[[0, 1, 2]], q[[0, 2, 3]]], np.float32), 0)
        t = pkg.GpuPathTracer(0)
        t.set_tuning(mode=2)
        assert t.sync(s, pkg.RenderOptions(width=480, height=270, scene_camera=0,
                                           path_trace=pkg.PathTraceOptions(samples_per_pixel=4, max_bounces=4)))
        t.set_camera(eye=(0.0, 1.0, 3.0), target=(0.0, 0.0, 0.0), yfov=0.8)
        times = []
        for _ in range(4):
            t.reset()
            t.finish()
            t0 = time.perf_counter()
            t.refine(4)
            t.finish()
            times.append(time.perf_counter() - t0)
        best.append(min(times))
    assert best[1] < 8.0 * best[0], best
