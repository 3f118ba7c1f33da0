"""The warp-per-query kernel (csrc/pm_photonmap.cu) where tiles never answer: maps of
fewer photons than tiles take, of at most k photons, and k above the tiles' largest.
Neighbour lists are the oracle's, radiance within 1e-5 of FP64 sums over them (the
bound of test_knn_gpu.py)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from photon_mapping_b200 import PhotonMap
from photon_mapping_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [
    (1, 1), (1, 5), (7, 8), (8, 8), (9, 8), (50, 50), (49, 50), (51, 50), (300, 300),
    (300, 1024), (1024, 1024), (1025, 1024),
    (4095, 50), (4096, 50), (4095, 224), (4096, 225), (60_000, 448), (60_000, 449),
    (60_000, 1024)])
@pytest.mark.parametrize("kind", ("walls", "point"))
def test_lists_and_radiance(ctx, n, k, kind):
    ph = W.wall_photons(n, n + k)
    if kind == "point":  # all at one distance: the buffer is cut at every round
        ph[:, 3:6] = (0.25, 0.5, 0.75)
    pm = PhotonMap(ctx)
    pm.setPhotons(ph)
    pm.build()
    q = W.wall_queries(301, 3)
    q[5, 0] = np.nan
    q[6, 1] += 1e4
    idx, cnt, md2 = pm.query_knn(q[:, :3], k)
    oidx, ocnt, omd2 = O.knn(ph, q[:, :3], k)
    np.testing.assert_array_equal(cnt, ocnt)
    np.testing.assert_array_equal(idx, oidx)
    np.testing.assert_array_equal(md2, omd2)
    rgb = pm.radiance(q, k, n)
    want = O.radiance_fp64(ph, oidx, ocnt, omd2, q, n)
    ok = np.isfinite(want)
    assert (np.abs(rgb - want)[ok] <= 1e-5 * np.abs(want[ok])).all()
    # the same sums whatever radius and neighbour in the work item came first
    order = np.random.default_rng(1).permutation(301)
    np.testing.assert_array_equal(pm.radiance(q[order], k, n), rgb[order])
