"""vgb_first_hit_ids queued on a stream that does not wait for the default one: the instance table (which
travels with the launch up to 256 instances, and is copied for more) is in place when the kernel reads it."""
from __future__ import annotations

import numpy as np
import pytest

from vira_gb300 import Scene, capi
from vira_gb300.spectral import FOUR_BAND

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ninst", [256, 257, 5000])
def test_ids_on_a_side_stream(gpu, ninst):
    import torch

    scene = Scene(FOUR_BAND, device=0)
    lib, ctx = capi.load(), scene.context()
    n = 1 << 16
    per = 3
    side = torch.cuda.Stream()
    for turn in range(20):     # another table each time: a stale one gives other instances
        rng = np.random.default_rng(turn)
        inst, mesh = rng.permutation(ninst).astype(np.uint32), rng.integers(0, 99, ninst).astype(np.uint32)
        table = np.stack([per * np.arange(ninst, dtype=np.uint32), inst, mesh], 1).astype(np.uint32)
        ids = rng.integers(0, per * ninst, n)
        with torch.cuda.stream(side):
            tri = torch.from_numpy(ids.astype(np.int32)).cuda()
            out = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(3)]
            nc = torch.empty((3, n), device="cuda")
            capi.check(lib.vgb_first_hit_ids(ctx, side.cuda_stream, n, tri.data_ptr(), 0, capi.ptr(table), ninst, None,
                                             None, *[o.data_ptr() for o in out], nc.data_ptr()), ctx)
            got = [x.cpu().numpy() for x in (tri, *out)]
        want = [ids % per, inst[ids // per], mesh[ids // per], np.zeros(n)]
        for g, w in zip(got, want):
            assert np.array_equal(g.astype(np.int64), w.astype(np.int64)), turn
        assert not nc.cpu().numpy().any()
    scene.close()
