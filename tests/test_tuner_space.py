"""The autotuner's space: the NEE kernel is searched in both wavefront modes, and
no two plans of the space launch the same kernels but for the two modes."""
from __future__ import annotations

import importlib

import pytest

# variants that are one kernel (include/oxpt_diag.h)
EQUAL = {"shade_variant": {0, 1}, "trace_variant": {4, 5}, "nee_variant": ({0, 1}, {3, 4})}


def _tuner(pkg):
    return importlib.import_module("oxideav_render_vulkan_b200.tuner")


@pytest.mark.parametrize("mode", ["MODE_WAVEFRONT", "MODE_WAVEFRONT_SPLIT"])
def test_nee_variants_are_searched(pkg, mode):
    tuner, N = _tuner(pkg), pkg._native

    def cost(p):
        return (0.0 if p.mode == getattr(N, mode) else 5.0) + (0.0 if p.nee_variant == 2 else 1.0)
    log = []
    best = tuner.coordinate_descent(cost, log=log)
    assert best.mode == getattr(N, mode) and best.nee_variant == 2


def test_space_has_no_equal_variants(pkg):
    space = _tuner(pkg).SPACE
    for knob, pairs in EQUAL.items():
        for pair in pairs if isinstance(pairs, tuple) else (pairs,):
            assert len(pair & set(space[knob])) == 1, knob
