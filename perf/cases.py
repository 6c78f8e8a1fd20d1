"""The framework's working calls as measurable cases: single renders, path-traced frames, a batched
trajectory, adjoint passes, the rasterizer, ray batches and the chain after the film.

``listed()`` names fixed cases, ``draw(rng)`` gives one more of the same ranges, ``prepare(case,
seed)`` builds what a user's program holds before the call (scene, BVH, cameras, parameters),
``run(state)`` is one call through the public entry points, ``work(case)`` the bytes and operations
it cannot do without and ``exact(case, seed)`` the result in 64 bits where plain torch can form it.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

AU = 149597870700.0
SUN_RADIUS = 696000000.0
DEV = "cuda"


# ----------------------------------------------------------------------------- cases
def listed():
    return [
        # The smallest call: a thumbnail of a small terrain tile (the smoke render's size); launch
        # latency and host work are most of it.
        dict(name="direct_96px", kind="direct", posts=65, w=96, h=96, bands=4, spp=1, lens=False),
        # The plain direct-lighting frame of the benchmark: 0.52M triangles, 1024^2, 1 spp.
        dict(name="direct_1024px", kind="direct", posts=513, w=1024, h=1024, bands=4, spp=1, lens=False),
        # A camera as it is used in earnest, at the default 1920 x 1080: lens distortion, depth of
        # field, smooth shading, two lights, an ambient term, velocity and triangle-size passes, 3 bands.
        dict(name="direct_1080p_lens", kind="direct", posts=257, w=1920, h=1080, bands=3, spp=4, lens=True),
        # A small odd-sized path-traced preview, one band, denoised.
        dict(name="path_301x203_denoised", kind="path", posts=129, w=301, h=203, bands=1, spp=16, bounces=2, rr=0,
             tex=96, denoise=True),
        # A medium path-traced frame over a crater DEM of 2.1M triangles, 8 bands.
        dict(name="path_512px", kind="path", posts=1025, w=512, h=512, bands=8, spp=16, bounces=3, rr=2, tex=1024,
             denoise=False),
        # The benchmark's frame size and options over 8.4M triangles (the largest case).
        dict(name="path_2048px", kind="path", posts=2049, w=2048, h=2048, bands=8, spp=4, bounces=3, rr=2, tex=2048,
             denoise=False),
        # A descent trajectory of uneven frames in one batched call.
        dict(name="trajectory_15", kind="batch", posts=513, frames=15, maxres=1024, bands=8, maxspp=16),
        # One step of the albedo + height inversion: forward, backward and a second forward at the
        # candidate heights (the vertices move twice).
        dict(name="inversion_4x256px", kind="inversion", posts=513, res=256, views=4, spp=16, bounces=2, tex=512),
        # The fused forward + adjoint of many views of a smooth-shaded asteroid.
        dict(name="asteroid_12_views", kind="asteroid", subdiv=7, views=12, maxres=512, spp=8),
        # The rasterizer's preview of the crater DEM with lighting.
        dict(name="raster_1024px", kind="raster", posts=1025, w=1024, h=1024, bands=8, tex=1024),
        # Device-resident ray batches (range sensors, line-of-sight tests): scattered closest hits
        # and occlusion tests over a GPU-built tree.
        dict(name="rays_2m", kind="rays", posts=1025, rays=2000003),
        # The film's way to an image: 81^2 PSF on the received power, then the noisy sensor.
        dict(name="psf_sensor_1024px", kind="film", w=1024, h=1024, bands=4, psf=81),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["direct", "direct", "path", "path", "batch", "inversion", "asteroid", "raster", "rays", "film"])
    bands = rng.choice([1, 3, 4, 8])
    if kind == "direct":
        w, h = _log(rng, 64, 1600), _log(rng, 64, 1600)
        spp = max(1, min(_log(rng, 1, 16), 8000000 // (w * h)))
        return dict(kind=kind, posts=_log(rng, 33, 700), w=w, h=h, bands=bands, spp=spp, lens=rng.random() < 0.3)
    if kind == "path":
        w, h = _log(rng, 64, 1500), _log(rng, 64, 1500)
        spp = max(1, min(_log(rng, 1, 48), 4000000 // (w * h)))
        return dict(kind=kind, posts=_log(rng, 65, 1100), w=w, h=h, bands=bands, spp=spp, bounces=rng.randint(1, 4),
                    rr=rng.choice([0, 2]), tex=_log(rng, 32, 1024), denoise=rng.random() < 0.25)
    if kind == "batch":
        return dict(kind=kind, posts=_log(rng, 65, 600), frames=rng.randint(2, 15), maxres=_log(rng, 100, 1000),
                    bands=bands, maxspp=rng.choice([1, 4, 16]))
    if kind == "inversion":
        return dict(kind=kind, posts=_log(rng, 65, 700), res=_log(rng, 48, 300), views=rng.randint(1, 5),
                    spp=_log(rng, 2, 16), bounces=rng.randint(0, 2), tex=_log(rng, 32, 512))
    if kind == "asteroid":
        return dict(kind=kind, subdiv=rng.randint(4, 7), views=rng.randint(1, 12), maxres=_log(rng, 64, 512),
                    spp=_log(rng, 1, 8))
    if kind == "raster":
        return dict(kind=kind, posts=_log(rng, 65, 1100), w=_log(rng, 64, 1500), h=_log(rng, 64, 1500), bands=bands,
                    tex=_log(rng, 32, 1024))
    if kind == "rays":
        return dict(kind=kind, posts=_log(rng, 65, 1100), rays=_log(rng, 1000, 3000000))
    return dict(kind="film", w=_log(rng, 64, 1100), h=_log(rng, 64, 1100), bands=bands,
                psf=2 * _log(rng, 3, 40) + 1)


# ----------------------------------------------------------------------------- inputs
def _bands(n):
    from vira_gb300 import EIGHT_BAND, FOUR_BAND, SpectralBands

    return {4: FOUR_BAND, 8: EIGHT_BAND}.get(n) or SpectralBands.uniform(n, 400, 1000)


def _terrain(n, posting, seed, amp, craters):
    """n x n FP32 heights: fBm (Hurst 0.8) scaled to +-amp, with a field of parabolic craters."""
    g = torch.Generator().manual_seed(int(seed))
    m = 1 << max(3, (n - 1).bit_length())
    k = torch.fft.fftfreq(m, dtype=torch.float64).to(DEV)
    k = torch.sqrt(k[None, :] ** 2 + k[:, None] ** 2)
    k[0, 0] = math.inf
    z = torch.randn((2, m, m), generator=g).to(DEV).double()
    h = torch.fft.ifft2(torch.complex(z[0], z[1]) * k ** -1.8).real
    i = torch.arange(n, device=DEV) % m
    h = h[i][:, i]
    h = (h - h.min()) / (h.max() - h.min()) * (2 * amp) - amp
    if craters:
        size = (n - 1) * posting
        for u in torch.rand((120, 3), generator=g).tolist():
            d = min(2.0 * posting * (1.0 - 0.97 * u[2]) ** (-1 / 1.5) * 4, 0.12 * size)
            r = d / 2 / posting
            cx, cy, e = u[0] * (n - 1), u[1] * (n - 1), int(1.5 * r) + 1
            x0, x1, y0, y1 = max(0, int(cx) - e), min(n, int(cx) + e + 1), max(0, int(cy) - e), min(n, int(cy) + e + 1)
            xx = (torch.arange(x0, x1, device=DEV) - cx)[None, :] / r
            yy = (torch.arange(y0, y1, device=DEV) - cy)[:, None] / r
            q = torch.sqrt(xx * xx + yy * yy)
            bowl = 0.04 * d - 0.24 * d * (1 - q * q)
            rim = 0.04 * d * (1.5 - q) / 0.5
            h[y0:y1, x0:x1] += torch.where(q <= 1, bowl, torch.where(q <= 1.5, rim, torch.zeros_like(q)))
    return h.float().cpu().numpy()


def _textured(scene, heights, posting, tex, nb, seed):
    """A DEM mesh with a lognormal albedo texture (median 0.12, sigma 0.3) over its grid."""
    from vira_gb300 import Mesh, synthetic

    n = heights.shape[0]
    mesh = Mesh.from_dem(heights, posting, albedo=1.0, nbands=nb)
    mesh.uv = synthetic.grid_uvs(n, n, n)
    g = torch.Generator().manual_seed(int(seed) + 77)
    a = (0.12 * torch.exp(0.3 * torch.randn((tex, tex), generator=g))).numpy()
    mesh.albedo_map = np.ascontiguousarray(np.repeat(a[:, :, None], nb, axis=2))
    scene.new_instance(scene.add_mesh(mesh))
    return mesh


def _camera(w, h, pos, target, fov=30.0):
    from vira_gb300 import Camera

    cam = Camera()
    cam.set_resolution(w, h)
    cam.set_sensor_size(36.0 / 1000.0)
    cam.set_field_of_view(fov)
    cam.set_local_position(*[float(x) for x in pos])
    cam.look_at([float(x) for x in target])
    return cam


def _sun_dir(az_deg, el_deg):
    a, e = math.radians(az_deg), math.radians(el_deg)
    return np.array([math.cos(e) * math.cos(a), math.cos(e) * math.sin(a), math.sin(e)])


def _direct_setup(case, seed):
    """Heights, posting, camera pose, sun and albedo of a direct-lighting case (no framework code)."""
    r = np.random.default_rng(seed)
    posting = 5120.0 / (case["posts"] - 1)
    h = _terrain(case["posts"], posting, seed, 200.0, False)
    pos = np.array([r.normal(-1500.0, 50.0), r.normal(0.0, 50.0), 5000.0])
    return h, posting, pos, np.array([r.normal(0, 50), r.normal(0, 50), 0.0]), (float(r.uniform(0, 360)), 30.0), 0.12


def prepare(case, seed):
    from vira_gb300 import Mesh, Scene

    kind = case["kind"]
    s = dict(case)
    r = np.random.default_rng(seed + 1)
    if kind == "film":
        from vira_gb300 import sensor

        nb = case["bands"]
        scene = Scene(_bands(nb))
        g = torch.Generator(device=DEV).manual_seed(int(seed))
        p = torch.rand((nb, case["h"], case["w"]), generator=g, device=DEV)
        s["power"] = (2e-12 * p * p + 2e-9 * (p > 0.9999)).float()    # a lit scene with a few bright points
        sig = np.linspace(1.2, 2.0, nb) * (1 + 0.1 * r.random())
        psf = sensor.GaussianPSF(sig, 1.3 * sig, 20.0)
        s["kernel"] = psf.make_kernel(scene.bands, case["psf"], 2)
        s["sensor"] = sensor.SensorModel(simulate_photon_noise=True, seed=int(seed),
                                         noise_model=sensor.NoiseModelConfig(dark_current=20.0, readout_noise_std=3.0))
        s["scene"] = scene
        return s
    if kind == "asteroid":
        from vira_gb300 import workloads

        scene, views, _ = workloads.asteroid(subdivisions=case["subdiv"], lmax=8, nviews=case["views"],
                                             spp=case["spp"], seed=int(seed) % 100000)
        for i, v in enumerate(views):
            res = max(16, case["maxres"] * (4, 1, 2)[i % 3] // 4)
            v.camera.set_resolution(res, res)
        scene.build_tlas()
        s["targets"] = []
        g = torch.Generator(device=DEV).manual_seed(int(seed))
        for v in views:
            w, h = v.camera.resolution
            s["targets"].append(2.0 * torch.rand((scene.bands.size, h, w), generator=g, device=DEV))
        s["scene"], s["views"] = scene, views
        return s
    if kind == "inversion":
        from vira_gb300 import FOUR_BAND
        from vira_gb300.autograd import View

        scene = Scene(FOUR_BAND)
        posting = 5120.0 / (case["posts"] - 1)
        h = _terrain(case["posts"], posting, seed, 100.0, True)
        mesh = _textured(scene, h, posting, case["tex"], 4, seed)
        scene.new_sun(temperature=5778.0)
        s["views"] = []
        for v in range(case["views"]):
            az = 2 * math.pi * v / case["views"] + r.uniform(0, 1)
            cam = _camera(case["res"], case["res"], (500 * math.cos(az), 500 * math.sin(az), 2000.0), (r.normal(0, 100), r.normal(0, 100), 0.0))
            s["views"].append(View(camera=cam, sun_position=AU * _sun_dir(r.uniform(0, 360), 10 + 50 * (v + 1) / case["views"]), frame=v))
        o = scene.pathtracer.options
        o.samples, o.bounces, o.seed = case["spp"], case["bounces"], int(seed)
        scene.pathtracer.render_passes.simulate_lighting = True
        scene.build_tlas()
        z = mesh.positions[:, 2]
        s["texture"] = torch.from_numpy(mesh.albedo_map).to(DEV).requires_grad_(True)
        s["heights"] = torch.from_numpy(z.copy()).to(DEV).requires_grad_(True)
        s["candidate"] = torch.from_numpy(z + r.normal(0, 0.5, z.shape).astype(np.float32)).to(DEV)
        g = torch.Generator(device=DEV).manual_seed(int(seed))
        s["weight"] = torch.randn((case["views"], 4, case["res"], case["res"]), generator=g, device=DEV)
        s["scene"] = scene
        return s
    if kind == "rays":
        from vira_gb300 import FOUR_BAND, capi

        scene = Scene(FOUR_BAND)
        posting = 5120.0 / (case["posts"] - 1)
        scene.new_instance(scene.add_mesh(Mesh.from_dem(_terrain(case["posts"], posting, seed, 200.0, True), posting)))
        scene.bvh_options = capi.BvhOptions(0, 1, 0, 0)
        scene.build_tlas()
        g = torch.Generator(device=DEV).manual_seed(int(seed))
        n = case["rays"]
        o = torch.rand((n, 3), generator=g, device=DEV) * 4800 - 2400
        o[:, 2] = 400 + 200 * torch.rand(n, generator=g, device=DEV)
        d = torch.randn((n, 3), generator=g, device=DEV)
        d[:, 2] = -d[:, 2].abs() * 0.5
        s["o"], s["d"] = o, d / d.norm(dim=1, keepdim=True)
        s["tmax"] = 200 + 1800 * torch.rand(n, generator=g, device=DEV)
        s["scene"] = scene
        return s
    nb = case["bands"]
    scene = Scene(_bands(nb))
    sun = scene.new_sun(temperature=5778.0)
    pt = scene.pathtracer
    pt.options.seed = int(seed)
    pt.render_passes.simulate_lighting = True
    s["scene"] = scene
    if kind == "direct":
        h, posting, pos, target, (az, el), alb = _direct_setup(case, seed)
        mesh = Mesh.from_dem(h, posting, albedo=alb, nbands=nb)
        scene.new_instance(scene.add_mesh(mesh))
        scene.set_sun_direction(sun, azimuth_deg=az, elevation_deg=el)
        cam = _camera(case["w"], case["h"], pos, target)
        pt.options.samples = case["spp"]
        pt.options.deterministic_light = True
        if case["lens"]:
            pt.options.deterministic_light = False
            mesh.set_smooth_shading(True)
            lamp = scene.new_sphere_light(50.0, 100.0)
            scene[lamp].position = np.array([1000.0, -500.0, 2500.0])
            scene.set_ambient(0.02)
            cam.set_brown_distortion_coefficients(k1=-0.05, k2=0.01, p1=1e-4, p2=-2e-4)
            cam.enable_depth_of_field()
            cam.set_focus_distance(5000.0)
            pt.render_passes.save_velocity = pt.render_passes.save_triangle_size = True
            cam.velocity, cam.angular_rate = np.array([10.0, 0.0, -3.0]), np.array([0.0, 1e-3, 0.0])
        s["camera"] = cam
    elif kind in ("path", "raster"):
        posting = 10240.0 / (case["posts"] - 1)
        _textured(scene, _terrain(case["posts"], posting, seed, 200.0, True), posting, case["tex"], nb, seed)
        scene.set_sun_direction(sun, azimuth_deg=float(r.uniform(0, 360)), elevation_deg=30.0)
        s["camera"] = _camera(case["w"], case["h"], (r.normal(-2500, 50), r.normal(0, 50), 7000.0), (r.normal(0, 50), 0.0, 0.0))
        if kind == "path":
            pt.options.samples, pt.options.bounces, pt.options.rr_depth = case["spp"], case["bounces"], case["rr"]
            pt.options.denoise = case["denoise"]
        else:
            scene.rasterizer.render_passes.simulate_lighting = True
    else:
        from vira_gb300 import BatchFrame

        posting = 5120.0 / (case["posts"] - 1)
        scene.new_instance(scene.add_mesh(Mesh.from_dem(_terrain(case["posts"], posting, seed, 200.0, False), posting, albedo=0.12, nbands=nb)))
        s["frames"] = []
        for i, (res, spp) in enumerate(_frames(case)):
            t = i / max(1, case["frames"] - 1)
            alt = 20000.0 * (400.0 / 20000.0) ** t
            az = math.radians(40.0 * t + r.uniform(0, 5))
            g = 0.6 * alt * (1 - t)
            cam = _camera(res, res, (g * math.cos(az), g * math.sin(az), alt + 200.0), (r.normal(0, 100), r.normal(0, 100), 0.0))
            s["frames"].append(BatchFrame(camera=cam, samples=spp, frame=i, light_positions=[AU * _sun_dir(0.1 * i, 30.0)]))
    scene.build_tlas()
    return s


def _frames(case):
    """(resolution, samples) of each frame of a batched case: a fixed uneven mix."""
    r = np.random.default_rng(5)
    spps = [k for k in (1, 4, 16) if k <= case["maxspp"]]
    return [(max(16, int(case["maxres"] * r.choice([0.25, 0.5, 1.0]))), int(r.choice(spps))) for _ in range(case["frames"])]


# ----------------------------------------------------------------------------- the call
_PASSES = ("depth", "alpha", "albedo", "normal_global", "triangle_id", "received_power", "total_radiance",
           "direct_radiance", "indirect_radiance", "instance_id", "velocity_global", "velocity_camera", "triangle_size")


def _planes(rp):
    return {k: getattr(rp, k) for k in _PASSES if getattr(rp, k) is not None}


def run(s):
    kind, scene = s["kind"], s["scene"]
    if kind in ("direct", "path"):
        return _planes(scene.pathtracer.render(s["camera"], scene))
    if kind == "raster":
        return _planes(scene.rasterizer.render(s["camera"], scene))
    if kind == "batch":
        return scene.render_batch(s["frames"])
    if kind == "inversion":
        from vira_gb300.autograd import RenderViews

        img = RenderViews.apply(s["texture"], s["heights"], scene, s["views"])
        gt, gz = torch.autograd.grad((img * s["weight"]).sum(), [s["texture"], s["heights"]])
        with torch.no_grad():
            img2 = RenderViews.apply(s["texture"], s["candidate"], scene, s["views"])
        return {"image": img.detach(), "d_texture": gt, "d_heights": gz, "candidate": img2}
    if kind == "asteroid":
        from vira_gb300.autograd import render_adjoint_batch

        loss, rads, _, gp = render_adjoint_batch(scene, s["views"], s["targets"], torch.device(DEV, 0))
        return {"loss": loss, "radiance": rads, "d_positions": gp}
    if kind == "rays":
        from vira_gb300 import capi

        lib, ctx, n = capi.load(), scene.context(), s["rays"]
        tri = torch.empty(n, dtype=torch.int32, device=DEV)
        t = torch.empty(n, device=DEV)
        w = torch.empty((n, 3), device=DEV)
        occ = torch.empty(n, dtype=torch.int32, device=DEV)
        torch.cuda.current_stream().synchronize()
        o, d, tm = s["o"].data_ptr(), s["d"].data_ptr(), s["tmax"].data_ptr()
        capi.check(lib.vgb_trace_rays(ctx, o, d, None, n, 0, tri.data_ptr(), t.data_ptr(), w.data_ptr(), 1), ctx)
        capi.check(lib.vgb_trace_rays(ctx, o, d, tm, n, 1, occ.data_ptr(), None, None, 1), ctx)
        return {"triangle": tri, "t": t, "w": w, "occluder": occ}
    from vira_gb300 import sensor

    power = sensor.psf_convolve(scene, s["power"].clone(), s["kernel"])
    return {"power": power, "image": sensor.simulate_sensor(scene, power, s["sensor"])}


# ----------------------------------------------------------------------------- what a pass needs
def work(case):
    kind = case["kind"]
    if kind == "film":
        n = case["w"] * case["h"]
        taps = case["bands"] * case["psf"] ** 2
        return {"bytes": 4 * n * (2 * case["bands"] + 1) + 4 * taps, "flops": 2 * n * taps}
    if kind == "asteroid":
        tris, verts = 20 * 4 ** case["subdiv"], 10 * 4 ** case["subdiv"] + 2
        pix = sum(max(16, case["maxres"] * (4, 1, 2)[i % 3] // 4) ** 2 for i in range(case["views"]))
        rays, out = 2 * pix * case["spp"], 4 * (pix * 8 + 3 * verts)
    else:
        verts, tris = case["posts"] ** 2, 2 * (case["posts"] - 1) ** 2
        if kind == "direct":
            pix = case["w"] * case["h"]
            rays, out = pix * case["spp"] * (3 if case["lens"] else 2), 4 * pix * (5 * case["bands"] + (14 if case["lens"] else 7))
        elif kind == "path":
            pix = case["w"] * case["h"]
            rays, out = pix * case["spp"] * 2 * (1 + 0.5 * case["bounces"]), 4 * pix * (5 * case["bands"] + 7)
        elif kind == "raster":
            pix = case["w"] * case["h"]
            rays, out = pix, 4 * pix * (5 * case["bands"] + 7)
        elif kind == "batch":
            fr = _frames(case)
            rays, out = sum(2 * r * r * p for r, p in fr), sum(4 * r * r * (2 * case["bands"] + 2) for r, _ in fr)
        elif kind == "inversion":
            pix = case["views"] * case["res"] ** 2
            rays, out = 3 * 2 * pix * case["spp"] * (1 + 0.5 * case["bounces"]), 4 * (pix * 12 + 4 * case["tex"] ** 2 + 2 * verts)
        else:
            rays, out = 2 * case["rays"], case["rays"] * (28 + 24)
    tex = 4 * case.get("tex", 0) ** 2
    # a ray descends at least one root-to-leaf path of two box tests a level and one triangle test
    return {"bytes": int(out + 32 * verts + 12 * tris + tex), "flops": int(rays * (2 * 24 * math.log2(tris) + 60))}


# ----------------------------------------------------------------------------- 64-bit results
def exact(case, seed):
    """The PSF's output, and small plain direct-lighting renders, in 64 bits; None elsewhere: brute
    force over every ray and triangle takes minutes there, and the sensor's Poisson draws and the
    sampled paths have no value in plain arithmetic."""
    if case["kind"] == "film":
        s = prepare(case, seed)
        k = torch.from_numpy(s["kernel"]).to(DEV).double()
        p, c = s["power"].double(), case["psf"] // 2
        H, W, n = case["h"], case["w"], case["psf"]
        f = torch.fft.rfft2(p, s=(H + n - 1, W + n - 1)) * torch.fft.rfft2(k.flip(1, 2), s=(H + n - 1, W + n - 1))
        return {"power": torch.fft.irfft2(f, s=(H + n - 1, W + n - 1))[:, c:c + H, c:c + W], "image": None}
    if case["kind"] != "direct" or case["lens"] or case["spp"] != 1:
        return None
    if 2 * (case["posts"] - 1) ** 2 * case["w"] * case["h"] > 4e9:
        return None
    return _exact_direct(case, seed)


def _closest(o, d, v, tmax=None):
    """Closest hit (t, triangle, w1, w2) of FP64 rays against every triangle, by brute force."""
    a, e1, e2 = v[0], v[1] - v[0], v[2] - v[0]
    t_out = torch.full((o.shape[0],), math.inf, dtype=torch.float64, device=DEV)
    tri = torch.zeros(o.shape[0], dtype=torch.int64, device=DEV)
    b = torch.zeros((o.shape[0], 2), dtype=torch.float64, device=DEV)
    step = max(1, 4000000 // a.shape[0])
    for i in range(0, o.shape[0], step):
        oo, dd = o[i:i + step, None, :], d[i:i + step, None, :]
        p = torch.linalg.cross(dd, e2[None])
        det = (e1[None] * p).sum(-1)
        s = oo - a[None]
        u = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1[None])
        w = (dd * q).sum(-1) / det
        t = (e2[None] * q).sum(-1) / det
        t = torch.where((u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0), t, torch.full_like(t, math.inf))
        m, k = t.min(dim=1)
        j = torch.arange(k.shape[0], device=DEV)
        t_out[i:i + step], tri[i:i + step] = m, k
        b[i:i + step, 0], b[i:i + step, 1] = u[j, k], w[j, k]
    return t_out, tri, b


def _exact_direct(case, seed):
    h, posting, pos, target, (az, el), albedo = _direct_setup(case, seed)
    n, W, H = case["posts"], case["w"], case["h"]
    f64 = lambda x: torch.as_tensor(np.asarray(x, np.float32).astype(np.float64), device=DEV)   # noqa: E731
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)                                            # noqa: E731
    dot = lambda x, y: (x * y).sum(-1)                                                           # noqa: E731
    j, i = np.mgrid[0:n, 0:n]
    P = f64(np.stack([posting * (i - (n - 1) / 2), posting * ((n - 1) / 2 - j), h], -1).reshape(-1, 3))
    qi, qj = [x.T.ravel() for x in np.meshgrid(np.arange(n - 1), np.arange(n - 1), indexing="xy")]
    at = lambda x, y: x + y * n                                                                  # noqa: E731
    idx = np.stack([np.stack([at(qi, qj + 1), at(qi + 1, qj), at(qi, qj)], -1),
                    np.stack([at(qi + 1, qj), at(qi, qj + 1), at(qi + 1, qj + 1)], -1)], 1).reshape(-1, 3)
    idx = torch.from_numpy(idx.astype(np.int64)).to(DEV)
    v = [P[idx[:, k]] for k in range(3)]
    fn = unit(torch.linalg.cross(v[1] - v[0], v[2] - v[0]))
    vn = torch.zeros_like(P)
    for k in range(3):
        vn.index_add_(0, idx[:, k], fn)
    vn = unit(vn)
    # camera: pinhole through the pixel corners, 36 mm wide sensor, 30 degree field of view
    focal = 0.036 / 2 / math.tan(math.radians(30.0) / 2)
    zc = (target - pos) / np.linalg.norm(target - pos)
    xc = np.cross(-np.array([0.0, 0.0, 1.0]), zc)
    xc /= np.linalg.norm(xc)
    R = f64(np.stack([xc, np.cross(zc, xc), zc], 1))
    hx = lambda x, y: torch.stack([(x - W / 2) * 0.036 / W / focal, (y - H / 2) * 0.036 / W / focal, torch.ones_like(x)], -1)  # noqa: E731
    py, px = torch.meshgrid(torch.arange(H + 1, device=DEV).double(), torch.arange(W + 1, device=DEV).double(), indexing="ij")
    corner = unit(hx(px, py))
    d = unit(corner[:H, :W].reshape(-1, 3) @ R.T)
    o = f64(pos).expand_as(d)
    t, tri, b = _closest(o, d, v)
    hit = torch.isfinite(t)
    w = torch.stack([b[:, 0], b[:, 1], 1 - b[:, 0] - b[:, 1]], -1)
    ring = [idx[tri, 1], idx[tri, 2], idx[tri, 0]]
    X = sum(w[:, k:k + 1] * P[ring[k]] for k in range(3))
    N = fn[tri]
    sp = sum(w[:, k:k + 1] * (X - dot(X - P[ring[k]], vn[ring[k]])[:, None] * vn[ring[k]]) for k in range(3))
    X = torch.where((dot(sp - X, N) > 0)[:, None], sp, X)
    # off the surface by 256 units in the last place of each 32-bit coordinate
    ulp = torch.exp2(torch.floor(torch.log2(X.abs().clamp(min=1e-30))) - 23)
    X = torch.where(X.abs() < 1 / 32, X + N / 65536, X + torch.trunc(256 * N) * ulp)
    to = torch.from_numpy(AU * _sun_dir(az, el)).to(DEV) - X
    dist = to.norm(dim=-1)
    L = to / dist[:, None]
    st, _, _ = _closest(X, L, v)
    # 1 / pdf: the sun's solid angle, 2 pi (1 - sqrt(d^2 - r^2) / d) without cancellation
    q = torch.sqrt(dist ** 2 - SUN_RADIUS ** 2)
    pdf = 1 / (2 * math.pi * SUN_RADIUS ** 2 / (dist * (dist + q)))
    nl = dot(N, L).clamp(min=0)
    mis = pdf ** 2 / (pdf ** 2 + (nl / math.pi) ** 2)
    lit = torch.where(hit & ~torch.isfinite(st), albedo / math.pi * nl * nl * mis / pdf, torch.zeros_like(nl))
    rad = torch.stack([lit * b for b in _black_body(case["bands"], 5778.0)]).reshape(-1, H, W)
    # solid angle of a pixel's quadrilateral, and the aperture's area
    om = lambda a, b, c: 2 * torch.atan2(dot(a, torch.linalg.cross(b, c)), 1 + dot(a, b) + dot(b, c) + dot(c, a))   # noqa: E731
    c0, c1, c2, c3 = corner[:-1, :-1], corner[:-1, 1:], corner[1:, 1:], corner[1:, :-1]
    omega = om(c0, c1, c2).abs() + om(c0, c2, c3).abs()
    area = math.pi * (0.05 / 2.8 / 2) ** 2
    nan = torch.full_like(N, math.nan)
    alpha = hit.double()
    return {"depth": t.reshape(H, W), "alpha": alpha.reshape(H, W),
            "albedo": (albedo * alpha).reshape(1, H, W).expand(case["bands"], H, W).contiguous(),
            "normal_global": torch.where(hit[:, None], N, nan).T.reshape(3, H, W).contiguous(),
            "triangle_id": None, "received_power": rad * omega[None] * area, "total_radiance": rad,
            "direct_radiance": rad, "indirect_radiance": torch.zeros_like(rad), "instance_id": None}


def _black_body(n, temperature):
    """Planck's law over each band, the trapezoid rule on 1000 points."""
    nm = [(400, 500), (500, 600), (600, 700), (800, 900)] if n == 4 else [(400 + 600 * k / n, 400 + 600 * (k + 1) / n) for k in range(n)]
    c, h, kb = 299792458.0, 6.62607015e-34, 1.380649e-23
    out = []
    for lo, hi in nm:
        x = np.linspace(lo * 1e-9, hi * 1e-9, 1000)
        out.append(float(np.trapezoid(2 * h * c * c / x ** 5 / np.expm1(h * c / (x * kb * temperature)), x)))
    return out
