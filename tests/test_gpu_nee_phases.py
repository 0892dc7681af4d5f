"""split_nee's phases (environment, emissive triangles, punctual lights) where
their lists and tables change form: no sampled light, only one kind, more
punctual lights than visibility bits (32) and than the shared-memory table
(64), light strategies, vertex- and job-major, plain and batched. The phases
compute what the oracle computes, so accumulators are equal bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(pkg, punctual, emissive):
    s = pkg.Scene()
    m = s.add_material(pkg.material(base_color=(0.7, 0.6, 0.5, 1.0), double_sided=1))
    glass = s.add_material(pkg.material(base_color=(0.9, 0.95, 1.0, 1.0), transmission=0.8, roughness=0.2))
    lamp = s.add_material(pkg.material(emissive=(4.0, 3.0, 2.0)))
    r = np.random.default_rng(7)
    p = r.uniform(-1, 1, (120, 1, 3)) + r.uniform(-0.3, 0.3, (120, 3, 3))
    s.add_mesh(p[:80].astype(np.float32), m)
    s.add_mesh(p[80:].astype(np.float32), glass)
    if emissive:
        s.add_mesh((p[:emissive] * 0.5 + (0.0, 1.2, 0.0)).astype(np.float32), lamp)
    for k in range(punctual):
        a = 2.4 * k
        s.add_light(k % 3, position=(2 * np.cos(a), 1.0 + 0.02 * k, 2 * np.sin(a)),
                    direction=(-np.cos(a), -0.6, -np.sin(a)), intensity=1.0 + 0.1 * (k % 5), range=float(k % 4) * 3.0,
                    inner_cone=0.3, outer_cone=0.9)
    s.add_camera((1.2, 1.0, 3.2), (0.0, 0.2, 0.0), 0.9)
    return s


CASES = [(0, 0, False, 0), (0, 5, False, 0), (0, 0, True, 0), (1, 5, True, 0), (3, 5, True, 2), (3, 5, True, 1),
         (31, 2, True, 0), (32, 2, True, 0), (64, 0, True, 0), (67, 2, False, 0)]


def _tracer(pkg, punctual, emissive, sky, strategy, **tuning):
    t = pkg.GpuPathTracer(0)
    if sky:
        t.set_environment(pkg.EnvironmentMap.sky(64, 32))
    t.set_tuning(**tuning)
    assert t.sync(_scene(pkg, punctual, emissive), pkg.RenderOptions(
        width=33, height=27, path_trace=pkg.PathTraceOptions(samples_per_pixel=3, max_bounces=5,
                                                             strategy=pkg.LightStrategy(strategy))))
    return t


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("mode,nee", [(1, 3), (2, 1), (2, 5)])
def test_nee_phases_bit_exact(pkg, oracle, case, mode, nee):
    t = _tracer(pkg, *case, mode=mode, nee_variant=nee, wave_slots=500)
    t.refine(3)
    t.finish()
    cpu, _ = oracle.render(t.prepared(), 3)
    assert np.array_equal(t.read_accum().view(np.uint32), cpu.view(np.uint32))


@pytest.mark.parametrize("nee", [1, 3])
def test_nee_phases_in_a_batch(pkg, oracle, nee):
    tracers = [_tracer(pkg, *c) for c in CASES]
    ex = pkg.GpuPathTracer(0)
    ex.set_tuning(mode=2, nee_variant=nee)
    pkg.refine_batch(tracers, 2, ex)
    for c, t in zip(CASES, tracers):
        t.finish()
        cpu, _ = oracle.render(t.prepared(), 2)
        assert np.array_equal(t.read_accum().view(np.uint32), cpu.view(np.uint32)), c
