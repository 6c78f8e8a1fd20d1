"""Scenes of stellar size (coordinates from 1e9 on) and rays parallel to the axes: a direction component
of 0 must not let the reciprocal's product with a box's distance overflow and cull a box that holds the ray."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_wide_nodes import _check
from vira_gb300 import Camera, Mesh, Scene, capi, synthetic
from vira_gb300.spectral import FOUR_BAND

pytestmark = pytest.mark.gpu
F = np.float32


def _scene(posting, layout=0, builder=0):
    s = Scene(FOUR_BAND, device=0)
    z = synthetic.fbm_heights(33, 0.8, seed=3, lo=-0.1 * posting, hi=0.1 * posting)
    s.new_instance(s.add_mesh(Mesh.from_dem(z, posting)))
    s.bvh_options = capi.BvhOptions(0, builder, 0, layout)
    return s


@pytest.mark.parametrize("builder", [0, 1], ids=["sah", "lbvh"])
@pytest.mark.parametrize("posting", [1e7, 1e8, 1e10], ids=str)
def test_closest_hits_of_a_stellar_scene(gpu, posting, builder):
    s = _scene(posting, builder=builder)
    s.build_tlas()
    _check(s, np.random.default_rng(5))
    s.close()


def test_camera_along_an_axis(gpu):
    """A camera that looks straight down: its middle row and column have a direction component of 0.
    The 8-wide layout, whose boxes are tested in another form, sees the same triangles."""
    got = []
    for layout in (0, 8):
        s = _scene(1e8, layout)
        sun = s.new_sun(temperature=5778.0)
        s.set_sun_direction(sun, azimuth_deg=30.0, elevation_deg=40.0)
        cam = Camera()
        cam.set_resolution(48, 32)
        cam.set_sensor_size(36.0 / 1000.0)
        cam.set_field_of_view(20.0)
        cam.set_local_position(3.0e7, 2.0e7, 6.0e9)
        cam.rotation = np.diag([1.0, -1.0, -1.0])
        s.pathtracer.render_passes.simulate_lighting = True
        rp = s.pathtracer.render(cam, s)
        got.append({k: getattr(rp, k).cpu().numpy() for k in ("triangle_id", "alpha", "total_radiance", "depth")})
        s.close()
    assert (got[0]["alpha"] == 1.0).all()
    for k in got[0]:
        assert np.array_equal(got[0][k].view(np.uint32), got[1][k].view(np.uint32)), k
