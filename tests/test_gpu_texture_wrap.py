"""Texture coordinates that wrap at the edges of the index arithmetic, against
the CPU oracle bit for bit: texture sides of 1, of no power of two and of
different width and height, coordinates far below zero and far above one, each
wrap mode, with one and with two filtered levels."""
from __future__ import annotations

import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wrap", [(0, 1), (1, 2), (2, 0)])
@pytest.mark.parametrize("size", [(1, 1), (1, 7), (5, 3), (37, 64)])
@pytest.mark.parametrize("shift", [-1.0e5, -2.5, 0.0])
def test_wrapped_taps(pkg, oracle, wrap, size, shift):
    rng = np.random.default_rng(size[0] * 100 + size[1])
    s = pkg.Scene()
    img = np.ones((size[1], size[0], 4), np.float32)
    img[..., :3] = rng.random((size[1], size[0], 3))
    t = s.add_texture(img, wrap=wrap, mag_linear=True, min_filter=5)
    m = pkg.material(base_color=(1, 1, 1, 1), metallic=0.0, roughness=0.7, tex={scenes.SLOT_BASE: (t, 0)})
    floor = scenes.quad_tris((-4, 0, 4), (4, 0, 4), (4, 0, -4), (-4, 0, -4))
    uv = np.array([[0, 3, 3, 3, 3, 0], [0, 3, 3, 0, 0, 0]], np.float32) + np.float32(shift)
    s.add_mesh(floor, s.add_material(m), uv0=uv)
    s.add_light(0, direction=(-0.3, -1.0, -0.4), intensity=2.5)
    s.add_camera((0.0, 0.9, 4.0), (0.0, 0.3, 0.0), 0.9)
    opts = pkg.RenderOptions(width=48, height=32, path_trace=pkg.PathTraceOptions(samples_per_pixel=2, max_bounces=3))
    tracer = pkg.GpuPathTracer(0)
    tracer.set_tuning(mode=pkg._native.MODE_WAVEFRONT_SPLIT)
    assert tracer.sync(s, opts)
    tracer.refine(2)
    tracer.finish()
    want, _ = oracle.render(tracer.prepared(), 2)
    got = tracer.read_accum()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
