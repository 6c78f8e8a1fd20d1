"""vgb_first_hit_ids against the same arithmetic in numpy: few instances (the table travels with the
launch), the last count that does, and one more; instances without triangles; misses."""
from __future__ import annotations

import numpy as np
import pytest

from vira_gb300 import Scene, capi
from vira_gb300.spectral import FOUR_BAND

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("first", [0, 1])
@pytest.mark.parametrize("ninst,npix", [(1, 1), (3, 1000), (256, 4097), (257, 70001)])
def test_ids_and_camera_normals(gpu, ninst, npix, first):
    import torch

    rng = np.random.default_rng(ninst + npix)
    counts = rng.integers(0, 50, ninst)
    counts[0] = 7
    starts = np.concatenate([[0], np.cumsum(counts)[:-1]])
    table = np.stack([starts, rng.permutation(ninst) + 5, rng.integers(0, 9, ninst)], 1).astype(np.uint32)
    tri = rng.integers(0, counts.sum(), npix)
    miss = rng.random(npix) < 0.2
    ids = np.where(miss, 0xFFFFFFFF, tri + first).astype(np.uint32)
    nrm = rng.standard_normal((3, npix)).astype(F)
    R = rng.standard_normal((3, 3)).astype(F)
    scene = Scene(FOUR_BAND, device=0)
    lib, ctx = capi.load(), scene.context()
    for rot in (None, R):
        t = torch.from_numpy(ids.view(np.int32).copy()).cuda()
        n = torch.from_numpy(nrm).cuda()
        out = [torch.full((npix,), 99, dtype=torch.int32, device="cuda") for _ in range(3)]
        nc = torch.full((3, npix), 99.0, device="cuda")
        torch.cuda.synchronize()
        capi.check(lib.vgb_first_hit_ids(ctx, torch.cuda.current_stream().cuda_stream, npix, t.data_ptr(), first,
                                         capi.ptr(table), ninst, n.data_ptr(), capi.ptr(rot), *[o.data_ptr() for o in out],
                                         nc.data_ptr()), ctx)
        k = np.searchsorted(starts, tri, side="right") - 1
        want = [np.where(miss, -1, np.asarray(x, np.int64)) for x in (tri - starts[k] + first, table[k, 1], table[k, 2], 0 * tri)]
        for got, w in zip([t, *out], want):
            assert np.array_equal(got.cpu().numpy().astype(np.int64), w.astype(np.int64))
        exp = np.zeros((3, npix), F) if rot is None else np.stack(
            [(nrm[0] * R[r, 0] + nrm[1] * R[r, 1]) + nrm[2] * R[r, 2] for r in range(3)])
        assert np.array_equal(nc.cpu().numpy(), exp)
    scene.close()
