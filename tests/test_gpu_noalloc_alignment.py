"""oxpt_dispatch_noalloc with table words at any 4-byte boundary of the
caller's memory: the accumulator is that of an aligned buffer, bit for bit."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("words", [0, 1, 2, 3])
def test_tables_at_any_word(pkg, oracle, words):
    import torch

    N = pkg._native
    w, h = 48, 32
    p = pkg.prepare(scenes.materials_scene(pkg),
                    pkg.RenderOptions(width=w, height=h, path_trace=pkg.PathTraceOptions(samples_per_pixel=2)))
    dev = torch.device("cuda", 0)
    geom = torch.from_numpy(p.geom.view(np.int32)).to(dev)
    attrs = torch.from_numpy(p.attrs).to(dev)
    atlas = torch.from_numpy(p.atlas.view(np.int16)).to(dev)
    packed = torch.from_numpy(np.concatenate([np.zeros(words, np.int32), p.tables.view(np.int32)])).to(dev)
    accum = torch.zeros((h, w, 4), dtype=torch.float32, device=dev)
    scene = N.DeviceScene(geom.data_ptr(), p.geom.size, attrs.data_ptr(), p.attrs.size,
                          packed.data_ptr() + 4 * words, p.tables.size, atlas.data_ptr(), p.atlas_side, p.atlas_layers)
    stream = torch.cuda.current_stream(dev)
    params, frame = p.params, N.Frame(0, 2, 0, h)
    assert N.lib().oxpt_dispatch_noalloc(C.byref(scene), C.byref(params), C.byref(frame),
                                         C.c_void_p(accum.data_ptr()), C.c_void_p(stream.cuda_stream)) == N.OK
    torch.cuda.synchronize(dev)
    want, _ = oracle.render(p, 2)
    assert np.array_equal(accum.cpu().numpy().view(np.uint32), want.view(np.uint32))
