"""The order in which the map's radix sort (csrc/pm_sort.cuh) leaves photons of equal
keys: that of their numbers.

A neighbour list does not show it, being ordered by distance and number, but a
radiance sum does: it goes by the photons' places in the sorted map (the photon at
place p belongs to class p & 31; a class is summed in the order of its places, then
the classes by a fixed tree), and floats of very different size make every order
another sum."""
from __future__ import annotations

import numpy as np
import pytest

from photon_mapping_b200 import PhotonMap
from photon_mapping_b200 import workloads as W

pytestmark = pytest.mark.gpu

PI = 3.14159265359  # core.h:7


def class_sum(thr):
    """thr: (k, 3) float32 in the order of places, the first of class 0."""
    part = np.zeros((32, 3), np.float32)
    for p, t in enumerate(thr):
        part[p & 31] += t
    x = part
    for o in (8, 16, 1, 2, 4):
        x = x + x[np.arange(32) ^ o]
    return x[0]


@pytest.mark.parametrize("n,every", [(5000, 1), (5000, 7), (70_001, 131), (300_000, 601),
                                     (300_000, 37)])
def test_photons_of_one_place_keep_their_order(ctx, n, every):
    """Every `every`-th photon at the map's lowest corner (key 0: the first places), the
    others elsewhere. k <= 256 of them lie under one node of the tree, whose groups
    are met in the order of their places; across the input they span many tiles of
    the sort."""
    rng = np.random.default_rng(n + every)
    ph = W.wall_photons(n, n)
    ph[:, 3:6] = rng.uniform(0.5, 1.0, (n, 3))
    here = np.arange(0, n, every)
    ph[here, 3:6] = 0.0
    ph[:, 0:3] = (10.0 ** rng.uniform(-4, 4, (n, 3))).astype(np.float32)
    ph[:, 6:9] = (0.0, 1.0, 0.0)
    k = min(256, len(here))
    pm = PhotonMap(ctx, 0)
    pm.setPhotons(ph)
    pm.build()
    q = np.zeros((1, 12), np.float32)
    q[0, :3] = (0.0, -0.25, 0.0)  # all of them at one distance: the first k are kept
    q[0, 3] = q[0, 7] = q[0, 11] = 1.0
    q[0, 4:7] = q[0, 8:11] = (0.0, 1.0, 0.0)
    idx, cnt, md2 = pm.query_knn(q[:, :3], k)
    np.testing.assert_array_equal(np.sort(idx[0]), here[:k])
    got = pm.radiance(q, k, n)[0]
    total = class_sum(ph[here[:k], 0:3]).astype(np.float64)
    want = (total / (float(n) * (PI * PI) * float(md2[0]))).astype(np.float32)
    np.testing.assert_array_equal(got, want)
