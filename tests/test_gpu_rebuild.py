"""Rebuilds of a scene's tree in one context: buffers kept from the tree before (larger, smaller, of the other
builder or layout) hold the new tree's nodes."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from test_gpu_wide_nodes import _check, _dem
from vira_gb300 import Scene, capi
from vira_gb300.spectral import FOUR_BAND

pytestmark = pytest.mark.gpu


def test_trees_in_turn(gpu):
    s = Scene(FOUR_BAND, device=0)
    s.new_instance(s.add_mesh(_dem(40)))
    s.build_tlas()
    lib, ctx = capi.load(), s.context()
    rng = np.random.default_rng(1)
    for leaf, builder, layout in ((4, 0, 0), (1, 1, 0), (8, 1, 0), (0, 0, 8), (1, 0, 2), (0, 1, 0), (8, 0, 0)):
        capi.check(lib.vgb_bvh_build(ctx, C.byref(capi.BvhOptions(leaf, builder, 0, layout))), ctx)
        if layout != 8:
            _check(s, rng)
        s.update_positions(0, (s.meshes[0].positions + rng.normal(0, 5.0, s.meshes[0].positions.shape)).astype(np.float32))
        if layout != 8:
            _check(s, rng)
    s.close()
