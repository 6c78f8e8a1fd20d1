"""The routes a render takes (k_front and k_fold over chunks of samples, the lean direct-lighting launch)
against the wavefront kernels alone (the persistent switch keeps a render on them): every plane bit for
bit, at the sizes where a route begins, a chunk ends and a tile is ragged.  And the fused adjoint with and
without its hit records."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from helpers import same_bits_or_nan
from vira_gb300 import Mesh, Scene, capi, synthetic, workloads
from vira_gb300.spectral import SpectralBands

pytestmark = pytest.mark.gpu
F = np.float32

PLANES = ("total_radiance", "direct_radiance", "indirect_radiance", "received_power", "albedo", "normal_global",
          "depth", "alpha", "triangle_id", "velocity_global", "velocity_camera", "triangle_size")


def _scene(w, h, bands=3, lights=1, smooth=False, posts=49):
    s = Scene(SpectralBands.uniform(bands, 400, 1000), device=0)
    m = Mesh.from_dem(synthetic.fbm_heights(posts, 0.8, seed=3, lo=-300.0, hi=300.0), 60.0, albedo=0.3, nbands=bands)
    m.smooth_shading = smooth
    s.new_instance(s.add_mesh(m))
    for k in range(lights):
        s.set_sun_direction(s.new_sun(5000.0 + 500 * k), azimuth_deg=100.0 * k, elevation_deg=25.0)
    cam = workloads._camera(s, max(w, 2), 2600.0, 20.0, 55.0)      # wider than the terrain: sky in the corners
    s[cam].set_resolution(w, h)
    s.pathtracer.render_passes.simulate_lighting = True
    return s, cam


def _render(s, cam, wavefront):
    lib, ctx = capi.load(), s.context()
    capi.check(lib.vgb_set_wavefront_tuning(ctx, 1 if wavefront else 0, 0, 0), ctx)
    rp = s.pathtracer.render(s[cam], s)
    st = s.pathtracer.last_stats
    out = {k: getattr(rp, k).cpu().numpy().copy() for k in PLANES if getattr(rp, k) is not None}
    return out, (st.rays_closest, st.rays_shadow, st.hits_closest), st.kernel_launches


CASES = {
    # width, height, samples, bounces, bands, lights, options
    "one_pixel": (1, 1, 1, 0, 1, 1, {}),
    "ragged": (33, 7, 5, 2, 3, 2, dict(rr=1)),
    "no_lights": (40, 24, 3, 1, 3, 0, dict(ambient=0.1)),
    "background": (65, 31, 4, 2, 4, 1, dict(background=0.5, ambient=0.1, smooth=True)),
    "unlit": (50, 50, 3, 2, 8, 1, dict(unlit=True)),
    "passes": (49, 33, 6, 1, 3, 1, dict(passes=True)),
    "lens": (70, 41, 3, 1, 3, 1, dict(lens=True)),
    "two_chunks": (1500, 1201, 11, 1, 1, 1, dict(passes=True)),          # 9 samples fit, so 6 and 5
    "lean_one_sample": (512, 512, 1, 0, 4, 2, dict(background=0.5, passes=True)),
    "below_lean": (511, 512, 1, 0, 4, 2, dict(background=0.5, passes=True)),
    "lean_samples": (1025, 1023, 3, 0, 1, 1, dict(lens=True, ambient=0.1)),
    "lean_unlit": (513, 517, 1, 0, 3, 1, dict(unlit=True)),
}


@pytest.mark.parametrize("name", list(CASES))
def test_routes_give_the_wavefront_s_planes(gpu, name):
    w, h, spp, bounces, bands, lights, o = CASES[name]
    s, cam = _scene(w, h, bands, lights, o.get("smooth", False))
    pt, c = s.pathtracer, s[cam]
    pt.options.samples, pt.options.bounces, pt.options.rr_depth, pt.options.seed = spp, bounces, o.get("rr", 0), 11
    pt.render_passes.simulate_lighting = not o.get("unlit", False)
    if "background" in o:
        pt.options.show_background = True
        s.set_background_emission(o["background"])
    if "ambient" in o:
        s.set_ambient(o["ambient"])
    if o.get("passes"):
        pt.render_passes.save_velocity = pt.render_passes.save_triangle_size = True
        c.velocity = np.array([3.0, -2.0, 1.0])
    if o.get("lens"):
        c.set_brown_distortion_coefficients(k1=-0.1, k2=0.02, p1=1e-3)
        c.enable_depth_of_field()
        c.set_focus_distance(2500.0)
    got, counts, launches = _render(s, cam, False)
    want, wcounts, wlaunches = _render(s, cam, True)
    assert launches < wlaunches
    assert counts == wcounts
    assert set(got) == set(want)
    for k in got:
        assert same_bits_or_nan(got[k], want[k]) if got[k].dtype == F else np.array_equal(got[k], want[k]), k
    if w > 1:
        assert (got["triangle_id"] >= 0).any()
    s.close()


def test_scratch_grows_and_shrinks_between_routes(gpu):
    """Frames of different sizes, bands' worth of samples and routes through one context, in turn."""
    s, cam = _scene(64, 64)
    ref = {}
    for turn in range(2):
        for w, h, spp, b in ((64, 64, 2, 1), (301, 203, 7, 2), (16, 9, 1, 0), (600, 500, 1, 0), (128, 50, 40, 1)):
            s[cam].set_resolution(w, h)
            s.pathtracer.options.samples, s.pathtracer.options.bounces = spp, b
            got, _, _ = _render(s, cam, False)
            if turn == 0:
                ref[w, h] = got
            else:
                want, _, _ = _render(s, cam, True)
                for k in got:
                    assert np.array_equal(got[k].view(np.uint32), ref[w, h][k].view(np.uint32)), k
                    assert same_bits_or_nan(got[k], want[k]) if got[k].dtype == F else np.array_equal(got[k], want[k]), k
    s.close()


@pytest.mark.parametrize("spp,bounces", [(4, 0), (3, 2), (250, 1)], ids=["records", "bounces", "too_many_for_records"])
def test_fused_adjoint_replays_what_it_recorded(gpu, spp, bounces):
    """The loss, the radiance and the gradients of the fused pass equal the separate renders and adjoints.
    Gradients: sums of the same terms in another order; FP32 sums of n terms stay within n^0.5 2^-24 of
    their magnitude, far under 1e-4 here."""
    import torch

    from vira_gb300.autograd import adjoint_views, forward_views, render_adjoint_batch

    s, views = workloads.inversion(posts=33, tex=16, resolution=17, nviews=2, spp=spp, bounces=bounces)
    s.build_tlas()
    dev = torch.device("cuda", 0)
    imgs = forward_views(s, views, dev)
    g = torch.Generator(device=dev).manual_seed(1)
    targets = [i + torch.randn(i.shape, generator=g, device=dev) * i.mean() for i in imgs]
    loss, rads, gt, gp = render_adjoint_batch(s, views, targets, dev)
    for r, i in zip(rads, imgs):
        assert torch.equal(r, i)
    assert abs(loss - float(sum(((i.double() - t.double()) ** 2).sum() for i, t in zip(imgs, targets)))) <= 1e-6 * loss
    rt, rp = adjoint_views(s, views, [2.0 * (i - t) for i, t in zip(imgs, targets)], dev, positions=True)
    for a, b in ((gt, rt), (gp, rp)):
        assert float((a - b).norm()) <= 1e-4 * float(b.norm()) and float(b.norm()) > 0
    s.close()


def test_autotuned_shape_is_kept_and_retuned(gpu):
    s, frames = workloads.trajectory(nframes=3, posts=65, resolutions=(48,), spps=(2,))
    lib, ctx = capi.load(), s.context()
    a = s.render_batch(frames)
    v = [C.c_uint32(0) for _ in range(3)]
    for again in (frames, frames[:1]):
        b = s.render_batch(again)
        capi.check(lib.vgb_batch_tuning(ctx, *[C.byref(x) for x in v]), ctx)
        assert v[0].value in (64, 128, 256) and v[1].value > 0 and v[2].value > 0
        for x, y in zip(a, b):
            for k in x:
                assert np.array_equal(x[k].cpu().numpy().view(np.uint32), y[k].cpu().numpy().view(np.uint32)), k
    s.close()
