"""The adjoint of the estimates by tiles of sorted queries (csrc/pm_knn_tile.cu) for
small k, at sizes that are sure to take them, against the warp-per-query kernel, which
answers while statistics are on.

Tolerance as in test_grad_tile_gpu.py: every term of a gradient component is positive,
so a sum of m floats in any order is within m 2^-24 of itself; a photon's adjoint and
a block's sum have at most about a thousand terms: 1e-4 for the two sides together."""
from __future__ import annotations

import numpy as np
import pytest

from photon_mapping_b200 import differentiable as D
from photon_mapping_b200 import scene as S
from photon_mapping_b200.camera import Camera

pytestmark = pytest.mark.gpu

TILE_WORK = 2_500_000  # least queries x (k + 50) of sorted queries for tiles


@pytest.mark.parametrize("w,h,spp,k,fg", [(161, 160, 4, 50, 1), (255, 257, 2, 1, 1),
                                          (127, 129, 4, 2, 0), (101, 100, 4, 224, 1)])
def test_tiles_give_the_warp_kernels_gradient(ctx, w, h, spp, k, fg):
    cam = Camera(S.CAMERA["position"], S.CAMERA["forward"], S.CAMERA["fov"])
    r = D.DiffRenderer(ctx, S.cornell_box(0), cam, w, h, spp, 20000, k,
                       final_gathering_depth=fg, max_depth=100, n_gather=1, seed=11)
    a0, e0 = r.base()
    g = np.ones((h, w, 3), np.float32)
    out = []
    for warp in (False, True):
        ctx.set_stats(warp)
        try:
            img = r.forward(a0, e0)
            assert r.stats["queries_global"] * (k + 50) >= 1.2 * TILE_WORK
            ga, ge = r.backward(g)
        finally:
            ctx.set_stats(False)
        out.append((img, np.concatenate([np.asarray(ga), np.asarray(ge)[None]])))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert np.abs(out[1][1]).max() > 0
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=1e-4)
