"""The nearest photon alone (k = 1): a search radius without any photon tells nothing of
how far it is, and k = 1 meets such radii more than any other k. The searches must not
creep up to it."""
from __future__ import annotations

import numpy as np
import pytest

from photon_mapping_b200 import PhotonMap
from photon_mapping_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_tiles_answer_one_about_as_fast_as_two(ctx):
    """1M estimates from 3M photons: 1.2 times the time of k = 2 (12 times it when the
    radius crept up). The bound of 4 is far from both."""
    import torch
    n, nq = 3_000_000, 1_000_000
    pm = PhotonMap(ctx)
    pm.setPhotons(W.wall_photons(n, 1))
    pm.build()
    q = torch.from_numpy(W.wall_queries(nq, 2)).cuda()
    out = torch.empty((nq, 3), device="cuda")
    st = torch.cuda.current_stream()
    ms = {}
    for k in (1, 2):
        t = []
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            ctx.check(ctx.lib.pm_photonmap_radiance_device(
                ctx.handle, 0, q.data_ptr(), nq, k, n, out.data_ptr(), st.cuda_stream),
                "pm_photonmap_radiance_device")
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
        ms[k] = min(t)
    assert ms[1] < 4 * ms[2], ms


@pytest.mark.parametrize("n", (5000, 100_000, 1_000_000))
def test_one_scans_no_more_than_four(ctx, n):
    """Photon groups scanned per neighbour list, by the kernel's own counters: the
    nearest photon needs no more of them than the four nearest (68 against 9 in 1M
    photons when the radius crept up and the search fell back to the patch bound)."""
    pm = PhotonMap(ctx)
    pm.setPhotons(W.wall_photons(n, 1))
    pm.build()
    q = np.ascontiguousarray(W.wall_queries(20_000, 2)[:, :3])
    per = {}
    for k in (1, 4):
        ctx.get_stats(reset=True)
        ctx.set_stats(True)
        try:
            pm.query_knn(q, k)
        finally:
            ctx.set_stats(False)
        st = ctx.get_stats(reset=True)
        assert st["queries"] == len(q)
        per[k] = st["leaves"] / st["queries"]
    assert per[1] <= per[4], per
