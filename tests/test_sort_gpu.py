"""The radix sort under the map build (csrc/pm_sort.cuh) at the edges of its
tiles, warps and rounds: every photon is in the built map exactly once."""
from __future__ import annotations

import numpy as np
import pytest

from photon_mapping_b200 import PhotonMap
from photon_mapping_b200 import workloads as W

pytestmark = pytest.mark.gpu

SIZES = (2, 31, 33, 255, 257, 2047, 2048, 2049, 4097, 70_001)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ("distinct", "few", "equal"))
def test_every_photon_once(ctx, n, kind):
    """distinct: a search at each photon's own place finds that photon (whole
    numbers, so exactly at distance 0). few, equal: 3 or 1 sort keys in all, and
    the photons of one place come in the order of their numbers."""
    ph = W.wall_photons(n, n)
    rng = np.random.default_rng(n)
    if kind == "distinct":
        cell = rng.permutation(64 ** 3)[:n]
        ph[:, 3:6] = np.stack([cell // 4096, cell // 64 % 64, cell % 64], 1)
        k = 1
    else:
        ph[:, 3:6] = rng.integers(0, 3 if kind == "few" else 1, n)[:, None]
        k = min(n, 64)
    pm = PhotonMap(ctx, 0)
    pm.setPhotons(ph)
    pm.build()
    if kind == "distinct":
        idx, cnt, md2 = pm.query_knn(ph[:, 3:6], k)
        assert (cnt == 1).all() and (md2 == 0).all()
        np.testing.assert_array_equal(idx[:, 0], np.arange(n))
        return
    for v in range(3 if kind == "few" else 1):
        here = np.flatnonzero(ph[:, 3] == v)[:k]
        if not len(here):
            continue
        idx, cnt, md2 = pm.query_knn(np.full((1, 3), v, np.float32), len(here))
        assert md2[0] == 0.0
        np.testing.assert_array_equal(np.sort(idx[0, :cnt[0]]), here)
