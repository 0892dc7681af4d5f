"""Graph refines of a single tracer: the scene sits in the captured kernels'
arguments, the camera, seed and sample range in the frame record. Steps whose
camera or seed changed reuse the graph, steps whose other options changed do
not, and every step equals the host-driven loop's bit for bit."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _steps(pkg):
    base = dict(samples_per_pixel=8, max_bounces=6)
    cams = [((0.3, 0.4, 3.0), False), ((2.0, 1.0, 1.5), False), ((0.0, 0.5, 6.0), True)]
    yield "same", cams[0], base
    for cam in cams:
        yield "same", cam, base
    yield "same", cams[1], dict(base, seed=77)
    yield "other", cams[1], dict(base, seed=77, strategy=pkg.LightStrategy.BSDF_ONLY)
    yield "other", cams[1], dict(base, seed=77, clamp=0.5)
    yield "other", cams[2], dict(base, max_bounces=3)


@pytest.mark.parametrize("mode", [1, 2])
def test_graph_steps_follow_camera_seed_and_options(pkg, mode):
    L = pkg._native.lib()
    scene = pkg.Scene.icosphere(freq=24, seed=2, n_materials=6, n_textures=3, tex_size=64, n_punctual=3, n_emissive=12,
                                material_mix=1)
    env = pkg.EnvironmentMap.sky(64, 32)
    tracers = []
    for graphs in (1, 0):
        t = pkg.GpuPathTracer(0)
        t.set_environment(env)
        t.set_tuning(mode=mode, graphs=graphs, wave_slots=700)
        tracers.append(t)
    builds, before = C.c_uint64(), None
    for what, (eye, ortho), pt in _steps(pkg):
        frames = []
        for t in tracers:
            t.sync(scene, pkg.RenderOptions(width=45, height=31, path_trace=pkg.PathTraceOptions(**pt)))
            t.set_camera(eye=eye, target=(0.0, 0.0, 0.0), yfov=0.9, orthographic=ortho, ymag=1.2)
            t.refine(2)
            t.refine(2)
            t.finish()
            frames.append(t.read_accum())
        assert np.array_equal(frames[0].view(np.uint32), frames[1].view(np.uint32)), (what, eye, pt)
        assert L.oxpt_diag_graph_builds(tracers[0].ctx, C.byref(builds)) == 0
        if before is not None:
            assert (builds.value == before) == (what == "same"), (what, eye, pt)
        before = builds.value
