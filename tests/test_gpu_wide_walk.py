"""The wide traversal kernels (csrc/wide_walk.cu) where they could part from
the reference walk: equal distances, boxes without thickness, trees of one
leaf, slivers and degenerate triangles, coordinates far from the origin,
axis-aligned rays, and several such scenes in one batch. Accumulators equal
the oracle's bit for bit (the walks are exact, so there is no tolerance)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(n, y=0.0, size=2.0):
    """n x n quads of two triangles in the plane y (boxes without thickness)."""
    c = np.linspace(-size / 2, size / 2, n + 1, dtype=np.float32)
    out = []
    for i in range(n):
        for j in range(n):
            p = [(c[i], y, c[j]), (c[i], y, c[j + 1]), (c[i + 1], y, c[j + 1]), (c[i + 1], y, c[j])]
            out += [[p[0], p[1], p[2]], [p[0], p[2], p[3]]]
    return np.asarray(out, np.float32)


def _soup(n, seed, size=0.3, centre=0.0, scale=1.0):
    r = np.random.default_rng(seed)
    p = r.uniform(-1, 1, (n, 1, 3)) + r.uniform(-size, size, (n, 3, 3))
    return (p * scale + centre).astype(np.float32)


def _scene(pkg, which):
    s = pkg.Scene()
    m = s.add_material(pkg.material(base_color=(0.7, 0.6, 0.5, 1.0), double_sided=1))
    m2 = s.add_material(pkg.material(base_color=(0.2, 0.6, 0.9, 1.0)))
    eye, target, kw = (1.5, 2.0, 3.0), (0.0, 0.0, 0.0), {}
    if which == "coincident":      # every hit has an equal one
        g = _grid(6)
        s.add_mesh(g, m)
        s.add_mesh(g[::-1].copy(), m2)
        s.add_mesh(_soup(60, 1), m)
    elif which == "layers":        # hits a few units in the last place apart
        for k in range(8):
            s.add_mesh(_grid(5, y=np.float32(0.5) + np.float32(k) * np.float32(2.0 ** -23)), m if k % 2 else m2)
    elif which == "slivers":
        t = _soup(300, 2)
        t[::3, 2] = t[::3, 1] + (t[::3, 0] - t[::3, 1]) * np.float32(1e-5)
        t[1::9, 2] = t[1::9, 1]
        t[2::9] *= np.float32(40.0)
        s.add_mesh(t, m)
    elif which == "far":           # the scene 3000 units from the origin
        s.add_mesh(_soup(400, 3, centre=3000.0), m)
        eye, target = (3002.0, 3002.0, 3004.0), (3000.0, 3000.0, 3000.0)
    elif which == "distant eye":   # a small scene seen from far away
        s.add_mesh(_soup(400, 4, scale=0.01), m)
        eye, kw = (0.0, 50.0, 0.0), dict(up=(0, 0, 1))
    elif which == "axis":          # rays along an axis, boxes without thickness
        s.add_mesh(_grid(9), m)
        s.add_mesh(_grid(4, y=0.75, size=1.0), m2)
        eye, kw = (0.0, 4.0, 0.0), dict(up=(0, 0, 1), orthographic=True, ymag=1.1)
    else:                          # trees of one leaf and a little more
        s.add_mesh(_soup(int(which), 5, size=1.5), m)
    s.add_camera(eye, target, 0.02 if which == "distant eye" else 0.9, **kw)
    s.add_light(0, direction=(0.3, -1.0, 0.2), intensity=3.0)
    s.add_light(1, position=tuple(np.add(target, (0.5, 1.5, 0.5))), intensity=5.0)
    return s


WHICH = ["coincident", "layers", "slivers", "far", "distant eye", "axis", "1", "2", "8", "9", "33"]


def _tracer(pkg, which, **tuning):
    t = pkg.GpuPathTracer(0)
    t.set_environment(pkg.EnvironmentMap.sky(32, 16))
    t.set_tuning(mode=2, **tuning)
    assert t.sync(_scene(pkg, which), pkg.RenderOptions(width=37, height=29, path_trace=pkg.PathTraceOptions(
        samples_per_pixel=4, max_bounces=6)))
    return t


@pytest.mark.parametrize("which", WHICH)
@pytest.mark.parametrize("variant,stack,refill", [(4, 0, 8), (3, 64, 32), (5, 0, 1)])
def test_wide_walk_bit_exact(pkg, oracle, which, variant, stack, refill):
    t = _tracer(pkg, which, trace_variant=variant, stack=stack, refill=refill)
    t.refine(4)
    t.finish()
    cpu, _ = oracle.render(t.prepared(), 4)
    assert np.array_equal(t.read_accum().view(np.uint32), cpu.view(np.uint32))


@pytest.mark.parametrize("graphs", [0, 1])
def test_wide_walk_in_a_batch(pkg, oracle, graphs):
    tracers = [_tracer(pkg, w) for w in WHICH]
    ex = pkg.GpuPathTracer(0)
    ex.set_tuning(mode=2, graphs=graphs, wave_slots=3000)
    pkg.pathtracer.refine_batch(tracers, 3, ex)
    for w, t in zip(WHICH, tracers):
        t.finish()
        cpu, _ = oracle.render(t.prepared(), 3)
        assert np.array_equal(t.read_accum().view(np.uint32), cpu.view(np.uint32)), w
