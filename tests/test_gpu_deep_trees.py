"""Trees deeper than the wide traversal's stack where they are folded by surface: nested clusters, each far
larger than the ones inside it and with nodes of its own, so that the fold shortens no chain.  Closest hits
against every triangle tested without a tree."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_wide_nodes import _check
from vira_gb300 import Mesh, Scene, capi
from vira_gb300.spectral import FOUR_BAND

pytestmark = pytest.mark.gpu


def _clusters(octaves, top):
    """Four triangles around a point 1.5 * 2^b from the origin on each axis, b from `top` down, and 64 at the origin;
    a triangle's box reaches 8 * 2^b about its point (less from axis to axis, so that every box is the larger one)."""
    c, h = [], []
    for k in range(octaves):
        e = 2.0 ** (top - k)
        for a in range(3):
            p = np.zeros(3)
            p[a] = e * (1.9 if k == 0 and a == 0 else 1.5)
            c += [p] * 4
            h += [8.0 * e * 2.0 ** (-a / 3)] * 4
    c += [np.zeros(3)] * 64
    h += [8.0 * 2.0 ** (top - octaves)] * 64
    v = np.array([[-1, 1, 0], [1, -1, -1], [0, 0, 1]], float)[None] * np.array(h)[:, None, None] + np.array(c)[:, None, :]
    p = v.reshape(-1, 3).astype(np.float32)
    return Mesh(positions=p, indices=np.arange(p.shape[0], dtype=np.uint32).reshape(-1, 3))


# binary / wide levels by surface / by height: 69 / 68 / 24 with either builder; by the host builder 246 / 245 / 83,
# which is rebuilt in Morton order: 73 / 71 / 26
@pytest.mark.parametrize("octaves,top,builder", [(21, 20, 0), (21, 20, 1), (80, 30, 0)], ids=["sah", "lbvh", "rebuilt"])
def test_deep_trees_find_every_closest_hit(gpu, octaves, top, builder):
    s = Scene(FOUR_BAND, device=0)
    s.new_instance(s.add_mesh(_clusters(octaves, top)))
    s.bvh_options = capi.BvhOptions(1, builder, 0, 0)
    s.build_tlas()
    _check(s, np.random.default_rng(octaves))
    if octaves == 21:
        m = s.meshes[0]
        s.update_positions(0, (m.positions * np.float32(1.25)).astype(np.float32))
        _check(s, np.random.default_rng(7))
    s.close()
