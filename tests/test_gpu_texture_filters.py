"""Every magnification and minification filter at the wrap edges of textures of
1 to 64 texels a side, against the CPU oracle bit for bit. The floor repeats
its texture 40 times towards the horizon, so that primary rays meet all mip
levels; bounced rays read the base level."""
from __future__ import annotations

import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wrap", [(0, 1), (2, 2)])
@pytest.mark.parametrize("size", [(1, 1), (7, 1), (5, 3), (37, 64)])
@pytest.mark.parametrize("mag_linear,min_filter", [(m, f) for m in (False, True) for f in range(6)])
def test_filters(pkg, oracle, mag_linear, min_filter, size, wrap):
    rng = np.random.default_rng(size[0] * 100 + size[1])
    s = pkg.Scene()
    img = np.ones((size[1], size[0], 4), np.float32)
    img[..., :3] = rng.random((size[1], size[0], 3))
    t = s.add_texture(img, wrap=wrap, mag_linear=mag_linear, min_filter=min_filter)
    m = pkg.material(base_color=(1, 1, 1, 1), metallic=0.0, roughness=0.7, tex={scenes.SLOT_BASE: (t, 0)})
    floor = scenes.quad_tris((-40, 0, 40), (40, 0, 40), (40, 0, -40), (-40, 0, -40))
    uv = np.array([[-20, -20, 20, -20, 20, 20], [-20, -20, 20, 20, -20, 20]], np.float32) + np.float32(0.5)
    s.add_mesh(floor, s.add_material(m), uv0=uv)
    s.add_light(0, direction=(-0.3, -1.0, -0.4), intensity=2.5)
    s.add_camera((0.0, 0.9, 4.0), (0.0, 0.3, 0.0), 0.9)
    opts = pkg.RenderOptions(width=40, height=32, path_trace=pkg.PathTraceOptions(samples_per_pixel=2, max_bounces=3))
    tracer = pkg.GpuPathTracer(0)
    tracer.set_tuning(mode=pkg._native.MODE_WAVEFRONT_SPLIT)
    assert tracer.sync(s, opts)
    tracer.refine(2)
    tracer.finish()
    want, _ = oracle.render(tracer.prepared(), 2)
    assert np.array_equal(tracer.read_accum().view(np.uint32), want.view(np.uint32))
