"""vgb_render with less memory than the samples in flight need: the allocator refuses, the frame goes in
smaller chunks of samples (down to the wavefront alone) and every plane is the same, call after call."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_front import PLANES, _scene
from vira_gb300 import capi
from vira_gb300.capi import VgbError

pytestmark = pytest.mark.gpu


def _render(s, cam):
    rp = s.pathtracer.render(s[cam], s)
    return {k: getattr(rp, k).cpu().numpy().copy() for k in PLANES if getattr(rp, k) is not None}, s.pathtracer.last_stats.kernel_launches


def _limit(s, nbytes):
    capi.check(capi.load().vgb_set_scratch_limit(s.context(), int(nbytes)), s.context())


@pytest.mark.parametrize("bounces", [0, 2])
def test_frames_fit_the_limit(gpu, bounces):
    s, cam = _scene(96, 64, bands=3, lights=2)
    s.pathtracer.render_passes.save_velocity = s.pathtracer.render_passes.save_triangle_size = True
    s.pathtracer.options.samples, s.pathtracer.options.bounces = 16, bounces
    want, launches = _render(s, cam)
    slots = 96 * 64
    most = 96 * 64 * 16 * 400        # more than a slot takes at 3 bands and 2 lights
    seen = [launches]
    for limit in (most, most / 4, most / 12, most / 20):
        _limit(s, limit)
        for _ in range(3):           # refused once, then rendered with what fits
            got, launches = _render(s, cam)
            for k in want:
                assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), (limit, k)
            seen.append(launches)
        assert len(set(seen[-3:])) == 1
    assert seen[0] == seen[1] and seen[-1] > seen[0]
    _limit(s, slots)                 # a byte a pixel: not even one sample
    for _ in range(2):
        with pytest.raises(VgbError) as e:
            _render(s, cam)
        assert e.value.status == 3
    _limit(s, 0)
    got, launches = _render(s, cam)
    assert launches == seen[0]
    for k in want:
        assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), k
    s.close()


def test_a_refused_allocation_does_not_fail_the_next_call(gpu):
    """What the allocator refused is reported by that call alone: the next one, of another kind, runs."""
    s, cam = _scene(64, 64)
    s.build_tlas()
    _limit(s, 1)
    with pytest.raises(VgbError):
        _render(s, cam)
    o = np.array([[0.0, 0.0, 5000.0]], np.float32)
    tri, _, _ = s.intersect(o, np.array([[0.0, 0.0, -1.0]], np.float32))
    assert tri[0] != capi.NO_HIT
    _limit(s, 0)
    _render(s, cam)
    s.close()


@pytest.mark.parametrize("w,h,samples,bounces,limits", [(1025, 1023, 1, 0, (1,)), (96, 64, 4, 1, (1.7e6, 2e6, 4e6))],
                         ids=["one_launch", "chunks"])
def test_no_memory_for_the_direction_table(gpu, w, h, samples, bounces, limits):
    """A camera with a lens distortion renders the same without its table of directions (one launch less
    where only the table was refused)."""
    s, cam = _scene(w, h, bands=3, lights=1)
    s[cam].set_brown_distortion_coefficients(k1=-0.05, k2=0.01, p1=1e-4, p2=-2e-4)
    s.pathtracer.options.samples, s.pathtracer.options.bounces = samples, bounces
    want, launches = _render(s, cam)
    for limit in limits:
        _limit(s, limit)
        for _ in range(2):
            got, n = _render(s, cam)
            for k in want:
                assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), (limit, k)
            assert bounces or n == launches - 1
    s.close()


def test_a_direct_frame_asks_for_no_path_state(gpu):
    """Without bounces a slot holds what the film asks for: at 3 bands 60 bytes with every sum of the
    path tracer's passes (radiance 12, state 4, direct 12, albedo 12, normal 12, depth 4, triangle 4)."""
    s, cam = _scene(128, 96, bands=3, lights=4)
    s.pathtracer.options.samples = 32
    _limit(s, 128 * 96 * 32 * 60)
    want, launches = _render(s, cam)
    assert launches == 2             # one chunk: k_front and k_fold
    _limit(s, 128 * 96 * 32 * 60 - 1)
    got, launches = _render(s, cam)
    assert launches > 2
    for k in want:
        assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), k
    s.close()


def test_scratch_makes_room_for_other_allocations(gpu):
    """An allocation of another call that the device refuses gives the render scratch back before it fails."""
    import torch

    s, cam = _scene(512, 511, bands=3, lights=1)
    s.pathtracer.options.samples, s.pathtracer.options.bounces = 16, 1
    want, _ = _render(s, cam)        # 4.2M slots of 176 bytes: 740 MB
    before = torch.cuda.mem_get_info()[0]
    one = torch.zeros(8, device="cuda")
    lib, ctx = capi.load(), s.context()
    # 2.9 TB of planes: refused before any of them is touched
    assert lib.vgb_psf_convolve(ctx, one.data_ptr(), 300000, 300000, 8, one.data_ptr(), 1, 1, 1) == 3
    assert torch.cuda.mem_get_info()[0] - before > 500e6
    got, _ = _render(s, cam)
    for k in want:
        assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), k
    s.close()
