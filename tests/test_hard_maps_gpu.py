"""Estimates from maps whose tree is of little use to tiles of queries (csrc/pm_knn_tile.cu):
photons far outside that leave all others in a few sort cells, most photons in one spot,
clusters of very different density. Results are those of the warp-per-query kernel
(which answers while statistics are on), and take about its time."""
from __future__ import annotations

import numpy as np
import pytest

from photon_mapping_b200 import PhotonMap
from photon_mapping_b200 import workloads as W

pytestmark = pytest.mark.gpu


def photons_of(kind, n):
    rng = np.random.default_rng(5)
    ph = W.uniform_photons(n, 1)
    if kind == "outliers":
        ph[:20, 3:6] *= 1e6
    elif kind == "spot":
        r = rng.normal(size=(n, 2)) * np.where(rng.uniform(size=(n, 1)) < 0.9, 0.002, 0.4)
        ph[:, 3], ph[:, 4], ph[:, 5] = 0.5 + r[:, 0], 0.0, 0.5 + r[:, 1]
    else:
        c = rng.integers(0, 50, n)
        ph[:, 3:6] = rng.uniform(0, 1, (50, 3))[c] + rng.normal(size=(n, 3)) * (
            10.0 ** rng.uniform(-5, -1, 50))[c, None]
    return ph


def queries_of(ph, nq, off):
    rng = np.random.default_rng(7)
    q = W.wall_queries(nq, 2)
    if off:
        q[:, :3] = rng.uniform(0, 1, (nq, 3))
    else:
        q[:, :3] = ph[rng.integers(0, len(ph), nq), 3:6] + rng.normal(size=(nq, 3)) * 1e-4
    return np.ascontiguousarray(q, np.float32)


def timed(ctx, q, k, n, out, repeat):
    import torch
    st = torch.cuda.current_stream()
    t = []
    for _ in range(repeat):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        ctx.check(ctx.lib.pm_photonmap_radiance_device(
            ctx.handle, 0, q.data_ptr(), q.shape[0], k, n, out.data_ptr(), st.cuda_stream),
            "pm_photonmap_radiance_device")
        b.record()
        torch.cuda.synchronize()
        t.append(a.elapsed_time(b))
    return min(t)


@pytest.mark.parametrize("kind,off,n,nq,k,slower", [
    # `slower`: bound of the time over the other kernel's (measured: 2.4 and 3.7 when
    # tiles tried on, 0.98 and 0.79 since they leave such queries early)
    ("outliers", True, 200_000, 60_000, 50, 1.7),
    ("clusters", False, 500_000, 150_000, 50, 1.7),
    ("spot", False, 200_000, 60_000, 200, None),
    ("spot", True, 20_000, 60_000, 448, None),
    ("clusters", True, 100_000, 300_000, 2, None),
])
def test_tiles_on_hard_maps(ctx, kind, off, n, nq, k, slower):
    import torch
    ph = photons_of(kind, n)
    pm = PhotonMap(ctx)
    pm.setPhotons(ph)
    pm.build()
    q = torch.from_numpy(queries_of(ph, nq, off)).cuda()
    out = [torch.full((nq, 3), -7.0, device="cuda") for _ in range(2)]
    ms = []
    for warp, o in zip((False, True), out):
        ctx.set_stats(warp)
        try:
            ms.append(timed(ctx, q, k, n, o, 3 if slower else 1))
        finally:
            ctx.set_stats(False)
    ctx.get_stats(reset=True)
    np.testing.assert_array_equal(out[0].cpu().numpy(), out[1].cpu().numpy())
    assert slower is None or ms[0] < slower * ms[1], ms


def test_radius_off_the_surfaces_does_not_overshoot(ctx):
    """Photon groups scanned per neighbour list at points off clustered photons, by the
    kernel's own counters: 1,459 when a radius grew up to 16-fold, 982 since it grows
    fourfold at most."""
    n, k = 500_000, 200
    ph = photons_of("clusters", n)
    pm = PhotonMap(ctx)
    pm.setPhotons(ph)
    pm.build()
    q = queries_of(ph, 20_000, True)
    ctx.get_stats(reset=True)
    ctx.set_stats(True)
    try:
        pm.query_knn(np.ascontiguousarray(q[:, :3]), k)
    finally:
        ctx.set_stats(False)
    st = ctx.get_stats(reset=True)
    assert st["leaves"] < 1200 * st["queries"], st
