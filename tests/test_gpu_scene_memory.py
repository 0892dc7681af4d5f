"""Device memory of scene builds that fail or that find no room: a failed build
leaves nothing allocated for a scene, and a build that has room only without
the scene before it takes that room."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from test_gpu_scene_prep import _Mesh, _Src

pytestmark = pytest.mark.gpu

NOMEM, INVALID = 2, 4
LAYER = 16384 * 16384 * 8  # bytes of the largest atlas layer


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _build(pkg, t, pos, layers=1, side=16384):
    mesh = _Mesh(len(pos), 0, pos.ctypes.data, None, None, None, None, None)
    src = _Src(C.addressof(mesh), 1, None, 0, None, 0, side, layers)
    ls, out = np.zeros(1, np.uint32), (C.c_uint32 * 3)()
    st = pkg._native.lib().oxpt_build_scene(t.ctx, C.byref(src), ls.ctypes.data, out)
    return st, list(out)


def _soup(n, seed=1):
    r = np.random.default_rng(seed)
    p = r.random((n, 3), np.float32)
    e = r.random((n, 6), np.float32) * np.float32(0.01)
    return np.concatenate([p, p + e[:, :3], p + e[:, 3:]], 1)


@pytest.mark.parametrize("why", [INVALID, NOMEM])
def test_failed_build_leaves_no_scene_memory(pkg, why):
    t = pkg.GpuPathTracer(0)
    pos = _soup(3000)
    assert _build(pkg, t, pos, side=64)[0] == 0  # loads the kernels, whose memory stays
    before = _free()
    assert _build(pkg, t, pos)[0] == 0
    held = before - _free()
    assert held > 0.9 * LAYER and t.memory()["scene"] > LAYER
    if why == INVALID:
        assert _build(pkg, t, pos, layers=0)[0] == INVALID
    else:
        assert _build(pkg, t, pos, layers=2000)[0] == NOMEM  # 4 TB
    assert t.memory()["scene"] == 0
    assert before - _free() < 0.1 * LAYER
    # the context still works
    scene = pkg.Scene.cornell()
    opts = pkg.RenderOptions(width=32, height=24, path_trace=pkg.PathTraceOptions(samples_per_pixel=2))
    fresh = pkg.GpuPathTracer(0)
    images = [x.render(scene, opts) for x in (t, fresh)]
    assert np.array_equal(*images)


def test_build_takes_the_old_scenes_room(pkg):
    """The scratch memory of the new scene does not fit beside the old one."""
    t = pkg.GpuPathTracer(0)
    assert _build(pkg, t, _soup(64), side=64)[0] == 0
    layers = (_free() - (1 << 30)) // LAYER
    assert _build(pkg, t, _soup(64), layers=layers)[0] == 0
    room = _free()
    assert room < 4 * LAYER
    pos = _soup(int(room * 1.1) // 240)  # 240 bytes of scratch a triangle, at least
    st, out = _build(pkg, t, pos, side=64)
    assert st == 0 and out[1] == len(pos)
    assert _free() > room + (layers - 8) * LAYER
