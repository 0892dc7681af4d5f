"""The cache network's kernels at the edges of their 128-sample tiles, against
the FP64 model with BF16 operands (oracle/nrc.py).

A gradient is compared by the norm of each layer. The device and the model
multiply the same BF16 numbers; what differs is the order of FP32 sums and,
rarely, a BF16 rounding that this flips (half a unit of 2^-8). Propagated
through four layers that stays below 3 % of the norm, for one sample as well
as for many. A prediction depends on its sample alone, so that the same sample
in a longer batch gives the same bits.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import nrc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 148 * 128 + 1, 2 * 148 * 128 + 65])
def test_tile_edges(pkg, n):
    L = pkg._native.lib()
    tracer = pkg.GpuPathTracer(0)
    h = C.c_void_p()
    assert L.oxpt_nrc_create(tracer.ctx, 11, C.byref(h)) == 0
    try:
        w = np.ascontiguousarray(nrc.init(21), np.float32)
        assert L.oxpt_nrc_set_weights(h, w.ctypes.data) == 0
        rng = np.random.default_rng(n)
        x = np.zeros((n + 150, 12), np.float32)
        x[:, :10] = rng.random((n + 150, 10))
        t = np.zeros((n, 4), np.float32)
        t[:, :3] = 0.2 + rng.random((n, 3))
        loss, g = C.c_float(), np.zeros(nrc.PARAMS, np.float32)
        assert L.oxpt_nrc_train(h, x.ctypes.data, t.ctypes.data, n, 0, C.byref(loss), g.ctypes.data) == 0
        want_loss, want = nrc.loss_grad(w, x[:n], t, bf=True)
        assert abs(loss.value - want_loss) <= 1e-2 * want_loss
        for l in range(nrc.LAYERS):
            a, b = g[nrc.OFFS[l]:nrc.OFFS[l + 1]], want[nrc.OFFS[l]:nrc.OFFS[l + 1]]
            assert np.linalg.norm(a - b) <= 0.03 * np.linalg.norm(b), l
        few, many = np.zeros((n, 4), np.float32), np.zeros((n + 150, 4), np.float32)
        assert L.oxpt_nrc_infer(h, x.ctypes.data, n, few.ctypes.data) == 0
        assert L.oxpt_nrc_infer(h, x.ctypes.data, n + 150, many.ctypes.data) == 0
        assert np.array_equal(few, many[:n])
    finally:
        L.oxpt_nrc_destroy(h)
