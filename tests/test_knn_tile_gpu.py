"""The tile kernel of sorted queries (csrc/pm_knn_tile.cu) against the
warp-per-query kernel and the FP64 oracle.

Both kernels keep the same photons and add them in the same order, so their
radiance is equal bit for bit; collecting search statistics selects the
warp-per-query kernel. The oracle bound is that of test_knn_gpu.py: 1e-5
relative against FP64 sums over exact neighbour sets.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from photon_mapping_b200 import PhotonMap
from photon_mapping_b200 import workloads as W

pytestmark = pytest.mark.gpu

def fewest(k):
    """The smallest number of unordered queries answered by tiles."""
    return -(-5_000_000 // (k + 50))


MIN_QUERIES = fewest(50)


def photons_of(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "walls":
        return W.wall_photons(n, seed)
    if kind == "cube":
        return W.uniform_photons(n, seed)
    if kind == "lattice":  # many equal distances, more than a bin holds
        return W.lattice_photons(int(round(n ** (1 / 3))), seed=seed)
    ph = W.uniform_photons(n, seed)
    if kind == "clusters":  # densities 1e6 apart, some photons far outside
        c = rng.integers(0, 50, n)
        ph[:, 3:6] = rng.uniform(0, 1, (50, 3))[c] + rng.normal(size=(n, 3)) * (
            10.0 ** rng.uniform(-5, -1, 50))[c, None]
        ph[:40, 3:6] *= 1e4
    elif kind == "point":  # no extent at all
        ph[:, 3:6] = (0.25, 0.5, 0.75)
    elif kind == "line":
        ph[:, 4:6] = 0.5
    return ph


def tile_and_warp(ctx, pm, q, k, n_emitted):
    import torch
    dq = torch.from_numpy(np.ascontiguousarray(q)).cuda()
    out = [torch.full((q.shape[0] + 1, 3), -7.0, device="cuda") for _ in range(2)]
    for i, o in enumerate(out):
        ctx.set_stats(i == 1)
        try:
            ctx.check(ctx.lib.pm_photonmap_radiance_device(
                ctx.handle, pm.map_id, dq.data_ptr(), q.shape[0], k, n_emitted, o.data_ptr(),
                torch.cuda.current_stream().cuda_stream), "pm_photonmap_radiance_device")
            torch.cuda.synchronize()
        finally:
            ctx.set_stats(False)
    ctx.get_stats(reset=True)
    assert all((o[-1] == -7.0).all() for o in out)
    return (o[:-1].cpu().numpy() for o in out)


@pytest.mark.parametrize("kind,n,more,k", [
    ("walls", 100_003, 0, 50),       # fewest queries
    ("walls", 100_003, -1, 50),      # one less: the other kernel
    ("walls", 4_096, 1, 1),          # fewest photons, ragged, k = 1
    ("walls", 4_101, 7, 8),          # last group of 5 photons
    ("cube", 200_000, 20_001, 100),
    ("cube", 60_000, 0, 448),        # largest k
    ("cube", 60_000, 0, 449),        # past it: the other kernel
    ("walls", 5_000, 0, 400),        # a large part of the map
    ("lattice", 27_000, 0, 64),
    ("clusters", 80_000, 9_999, 50),
    ("point", 5_000, 0, 20),
    ("line", 20_000, 0, 30),
    ("walls", 300_000, 600_000, 20),  # items of 32 queries
])
def test_tile_kernel_equals_warp_kernel(ctx, kind, n, more, k):
    nq = fewest(k) + more
    ph = photons_of(kind, n, 7)
    pm = PhotonMap(ctx)
    pm.setPhotons(ph)
    pm.build()
    q = W.wall_queries(nq, 8)
    rng = np.random.default_rng(9)
    if kind in ("cube", "clusters"):  # on and off the photons
        q[:, :3] = ph[rng.integers(0, ph.shape[0], nq), 3:6] + rng.normal(size=(nq, 3)) * 1e-3
    elif kind == "lattice":
        q[:, :3] = ph[rng.integers(0, ph.shape[0], nq), 3:6]
    q[rng.integers(0, nq, 40), 0] = np.nan
    q[rng.integers(0, nq, 40), 1] = np.inf
    q[rng.integers(0, nq, 40), :3] += 1e4  # far from every photon
    q[rng.integers(0, nq, 40), 4:7] *= -1  # wo below the surface
    got, want = tile_and_warp(ctx, pm, q, k, n)
    np.testing.assert_array_equal(got, want)
    part = rng.integers(0, nq, 200)
    part = part[np.isfinite(q[part, :3]).all(axis=1)]
    oidx, ocnt, omd2 = O.knn(ph, q[part, :3], k)
    fp64 = O.radiance_fp64(ph, oidx, ocnt, omd2, q[part], n)
    ok = np.isfinite(fp64)
    assert (np.abs(got[part] - fp64)[ok] <= 1e-5 * np.abs(fp64[ok])).all()


def test_estimates_in_flight_on_several_streams(ctx):
    """Calls on more streams than the context keeps query buffers for, none of
    them waited for: each equals the call on its own."""
    import torch
    pm = PhotonMap(ctx)
    pm.setPhotons(W.wall_photons(200_000, 1))
    pm.build()
    sizes = [MIN_QUERIES + 4096 * i for i in range(7)]
    qs = [torch.from_numpy(W.wall_queries(s, 20 + i)).cuda() for i, s in enumerate(sizes)]

    def call(q, out, stream):
        ctx.check(ctx.lib.pm_photonmap_radiance_device(
            ctx.handle, 0, q.data_ptr(), q.shape[0], 50, 200_000, out.data_ptr(),
            stream.cuda_stream), "pm_photonmap_radiance_device")

    want = []
    for q in qs:
        o = torch.empty((q.shape[0], 3), device="cuda")
        call(q, o, torch.cuda.current_stream())
        torch.cuda.synchronize()
        want.append(o)
    got = [torch.empty_like(o) for o in want]
    streams = [torch.cuda.Stream() for _ in qs]
    torch.cuda.synchronize()
    for _ in range(2):
        for q, o, s in zip(qs, got, streams):
            call(q, o, s)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_captured_estimate(ctx):
    """A call captured in a CUDA graph replays on new queries."""
    import torch
    pm = PhotonMap(ctx)
    pm.setPhotons(W.wall_photons(50_000, 1))
    pm.build()
    q = [torch.from_numpy(W.wall_queries(MIN_QUERIES, 30 + i)).cuda() for i in range(2)]
    dq, out = q[0].clone(), torch.empty((MIN_QUERIES, 3), device="cuda")

    def call(stream):
        ctx.check(ctx.lib.pm_photonmap_radiance_device(
            ctx.handle, 0, dq.data_ptr(), dq.shape[0], 50, 50_000, out.data_ptr(),
            stream.cuda_stream), "pm_photonmap_radiance_device")

    want = []
    for x in q:
        dq.copy_(x)
        call(torch.cuda.current_stream())
        torch.cuda.synchronize()
        want.append(out.clone())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(torch.cuda.current_stream())
    for x, w in zip(q, want):
        dq.copy_(x)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, w)
    del g
