"""Camera and light structs of the C ABI from what callers hand over: lists, arrays of either precision, torch
tensors, and sequences longer than what is used (an intrinsic inverse with a last row, a rate with a spare)."""
from __future__ import annotations

import numpy as np
import pytest

from vira_gb300 import Camera, Scene, capi
from vira_gb300.spectral import FOUR_BAND

F = np.float32


def _camera():
    c = Camera()
    c.set_resolution(20, 10)
    c.set_sensor_size(0.03)
    c.set_field_of_view(30.0)
    return c


@pytest.mark.parametrize("kind", ["list", "f64", "f32", "torch"])
def test_light_radiance_of_any_sequence(kind):
    import torch

    v = [0.1, 2.5, 1e-9, 7.0]
    s = Scene(FOUR_BAND)
    s.new_sphere_light(1.0, 2.0)
    s.lights[0].position = np.array([1.0, 2.0, 3.0])
    s.lights[0].radiance = {"list": v, "f64": np.array(v), "f32": np.array(v, F), "torch": torch.tensor(v, dtype=torch.float64)}[kind]
    arr, n = s.c_lights()
    assert n == 1
    assert np.array_equal(np.array(arr[0].radiance[:4], F), np.array(v, F))
    assert list(arr[0].radiance[4:]) == [0.0] * 4 and list(arr[0].position) == [1.0, 2.0, 3.0]


def test_camera_sequences_longer_than_used():
    c = _camera()
    want = bytes(c.to_c(np.zeros(3), 4, kinv=np.arange(6, dtype=F)))
    assert bytes(c.to_c(np.zeros(3), 4, kinv=[0, 1, 2, 3, 4, 5, 0, 0, 1])) == want
    c.velocity, c.angular_rate = [1.0, 2.0, 3.0, 9.0], np.array([4.0, 5.0, 6.0, 9.0])
    k = c.to_c(np.zeros(3), 4, kinv=np.arange(6, dtype=F))
    assert list(k.velocity) == [1.0, 2.0, 3.0] and list(k.angular_rate) == [4.0, 5.0, 6.0]
    c.distortion = (capi.DISTORTION_BROWN, [0.1, 0.2, 0.3, 0.4, 0.5])
    d = c.to_c(np.zeros(3), 4, kinv=np.arange(6, dtype=F)).distortion_coeffs
    assert np.array_equal(np.array(d[:5], F), np.array([0.1, 0.2, 0.3, 0.4, 0.5], F)) and list(d[5:]) == [0.0] * 7


def test_radiance_is_read_element_by_element():
    """Anything float() takes, element by element: a tensor whose memory numpy cannot see among it."""
    class Element:
        def __init__(self, x):
            self.x = x

        def __float__(self):
            return self.x

        def __array__(self, *a, **k):
            raise TypeError("not host memory")

    s = Scene(FOUR_BAND)
    s.new_sphere_light(1.0, 2.0)
    s.lights[0].position = np.zeros(3)
    s.lights[0].radiance = [Element(float(x)) for x in range(4)]
    arr, _ = s.c_lights()
    assert list(arr[0].radiance[:4]) == [0.0, 1.0, 2.0, 3.0]
