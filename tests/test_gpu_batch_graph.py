"""Captured batch launches (use_graph) after what they hold has changed: another mesh of the same frames,
moved vertices, another texture, another traversal limit."""
from __future__ import annotations

import numpy as np
import pytest

from vira_gb300 import Mesh, capi, synthetic, workloads
from vira_gb300.capi import VgbError

pytestmark = pytest.mark.gpu


def _same(s, frames, **kw):
    a, b = s.render_batch(frames, use_graph=True, **kw), s.render_batch(frames, use_graph=False, **kw)
    for x, y in zip(a, b):
        for k in x:
            assert np.array_equal(x[k].cpu().numpy().view(np.uint32), y[k].cpu().numpy().view(np.uint32)), k
    return np.concatenate([x["total_radiance"].cpu().numpy().ravel() for x in b])


@pytest.mark.parametrize("bounces", [0, 1])
def test_graph_follows_the_scene(gpu, bounces):
    s, frames = workloads.trajectory(nframes=3, posts=65, resolutions=(48,), spps=(2,))
    s.pathtracer.options.bounces = bounces
    seen = [_same(s, frames)]
    for posts, layout in ((40, 0), (90, 0), (66, 8), (65, 0)):         # smaller, larger, another layout
        z = synthetic.fbm_heights(posts, 0.8, seed=posts, lo=-300.0, hi=300.0)
        s.meshes[0] = Mesh.from_dem(z, 5120.0 / (posts - 1), albedo=0.3, nbands=s.bands.size)
        s.bvh_options = capi.BvhOptions(0, 0, 0, layout)
        s.mark_dirty()
        seen.append(_same(s, frames))
    s.update_positions(0, (s.meshes[0].positions + np.array([0, 0, 500.0], np.float32)).astype(np.float32))
    seen.append(_same(s, frames))
    for i, x in enumerate(seen):
        assert all(not np.array_equal(x, y) for y in seen[:i])
    lib, ctx = capi.load(), s.context()
    capi.check(lib.vgb_set_traversal_limit(ctx, 1), ctx)
    for graph in (True, False):
        with pytest.raises(VgbError) as e:
            s.render_batch(frames, autotune=False, use_graph=graph)
        assert e.value.status == 5
    capi.check(lib.vgb_set_traversal_limit(ctx, 0), ctx)
    assert np.array_equal(_same(s, frames, autotune=False), seen[-1])
    s.close()
