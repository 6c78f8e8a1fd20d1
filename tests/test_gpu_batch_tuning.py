"""When the batch autotuner times launch shapes again: not for the same kind of work on the same tree; for
another tree, size, sample count, number of lights or bounces; and after probes that gave up."""
from __future__ import annotations

import ctypes as C
import dataclasses

import pytest

from vira_gb300 import capi, workloads
from vira_gb300.capi import VgbError

pytestmark = pytest.mark.gpu
SHAPES = 6


def test_shapes_are_timed_once_per_kind_of_work(gpu):
    s, frames = workloads.trajectory(nframes=4, posts=65, resolutions=(48,), spps=(2,))
    lib, ctx = capi.load(), s.context()
    n = C.c_uint64(0)
    expect = 0

    def call(fr, timed):
        nonlocal expect
        s.render_batch(fr)
        expect += SHAPES if timed else 0
        capi.check(lib.vgb_batch_probes(ctx, C.byref(n)), ctx)
        assert n.value == expect

    call(frames, True)
    call(frames, False)
    call(frames[::-1], False)                                            # the same work in another order
    call([dataclasses.replace(f, samples=32) for f in frames], True)     # 16 times the samples
    call(frames, True)                                                   # the last kind is kept, no other
    call(frames[:1], True)                                               # a quarter of the tiles
    call(frames, True)
    s.pathtracer.options.bounces = 1
    call(frames, True)
    call(frames, False)
    s.new_sphere_light(50.0, 100.0)
    two = [dataclasses.replace(f, light_positions=[*f.light_positions, f.light_positions[0] * 0.5]) for f in frames]
    call(two, True)
    call(two, False)
    capi.check(lib.vgb_bvh_build(ctx, C.byref(capi.BvhOptions(0, 1, 0, 0))), ctx)
    call(two, True)
    capi.check(lib.vgb_bvh_build(ctx, C.byref(capi.BvhOptions(0, 0, 0, 0))), ctx)
    capi.check(lib.vgb_set_traversal_limit(ctx, 1), ctx)
    with pytest.raises(VgbError):
        s.render_batch(two)
    expect += SHAPES
    capi.check(lib.vgb_set_traversal_limit(ctx, 0), ctx)
    call(two, True)                                                      # nothing was kept of those
    call(two, False)
    s.close()
