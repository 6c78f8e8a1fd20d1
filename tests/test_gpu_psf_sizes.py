"""PSF convolution at every kernel width up to one past two groups of four taps (each width below 8 and each
remainder above has its own kernel), bit for bit against the oracle; widths and heights that differ."""
from __future__ import annotations

import numpy as np
import pytest

from vira_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,kh", [(1, 1), (2, 3), (3, 8), (4, 2), (5, 5), (6, 1), (7, 4), (8, 8), (9, 3), (10, 1), (11, 2), (127, 3)])
def test_every_width(gpu, kw, kh):
    import ctypes as C

    from oracle import oracle

    lib = capi.load()
    ctx = C.c_void_p()
    capi.check(lib.vgb_context_create(C.byref(ctx), 0))
    rng = np.random.default_rng(100 * kw + kh)
    img = rng.uniform(0, 1, (3, 37, 131)).astype(np.float32)
    img[0, 3, 5] = np.inf                     # a padded tap would make it a NaN
    kern = rng.uniform(0.1, 1, (3, kh, kw)).astype(np.float32)
    g = img.copy()
    capi.check(lib.vgb_psf_convolve(ctx, capi.ptr(g), 131, 37, 3, capi.ptr(kern), kw, kh, 0), ctx, "psf")
    assert np.array_equal(g.view(np.uint32), oracle.psf(img, kern).view(np.uint32))
    lib.vgb_context_destroy(ctx)
