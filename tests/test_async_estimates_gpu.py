"""pm_photonmap_radiance_device as an asynchronous call: many in flight, on one stream
and on several, beside a capture, and without memory for its query buffers."""
from __future__ import annotations

import numpy as np
import pytest

from photon_mapping_b200 import Context, PhotonMap
from photon_mapping_b200 import workloads as W

pytestmark = pytest.mark.gpu

N, K = 100_000, 50
MIN_QUERIES = 5_000_000 // (K + 50)  # fewest that tiles answer


@pytest.fixture
def own():
    """A context of its own: no query buffers yet."""
    with Context(0) as c:
        pm = PhotonMap(c)
        pm.setPhotons(W.wall_photons(N, 1))
        pm.build()
        yield c


def call(ctx, q, out, stream):
    ctx.check(ctx.lib.pm_photonmap_radiance_device(
        ctx.handle, 0, q.data_ptr(), q.shape[0], K, N, out.data_ptr(), stream.cuda_stream),
        "pm_photonmap_radiance_device")


def alone(ctx, q):
    import torch
    o = torch.empty((q.shape[0], 3), device="cuda")
    call(ctx, q, o, torch.cuda.current_stream())
    torch.cuda.synchronize()
    return o


def test_more_calls_in_flight_than_the_context_has_counters(own):
    import torch
    long_q = torch.from_numpy(W.wall_queries(8 * MIN_QUERIES, 2)).cuda()
    short = [torch.from_numpy(W.wall_queries(MIN_QUERIES + 999 * i, 3 + i)).cuda()
             for i in range(6)]
    long_want, want = alone(own, long_q), [alone(own, q) for q in short]
    first, others = torch.cuda.Stream(), [torch.cuda.Stream() for _ in short]
    long_got = [torch.zeros_like(long_want) for _ in range(80)]
    got = [[torch.zeros_like(w) for w in want] for _ in range(12)]
    torch.cuda.synchronize()
    for o in long_got:
        call(own, long_q, o, first)
    for row in got:
        for q, o, s in zip(short, row, others):
            call(own, q, o, s)
    torch.cuda.synchronize()
    assert all(torch.equal(o, long_want) for o in long_got)
    for row in got:
        assert all(torch.equal(o, w) for o, w in zip(row, want))


@pytest.mark.parametrize("mapped", (False, True))
def test_estimates_without_memory_for_query_buffers(own, mapped):
    """Little device memory left: the estimates take the kernel that needs none (with
    page-locked host buffers, which it reads and writes in place, or device ones)."""
    import torch
    nq = 4_000_000
    q = torch.from_numpy(W.wall_queries(nq, 7))
    dq = q.cuda()
    want = alone(own, dq)
    fill = []
    with Context(0) as c2:
        pm = PhotonMap(c2)
        pm.setPhotons(W.wall_photons(N, 1))
        pm.build()
        few = torch.empty((1000, 3), device="cuda")
        call(c2, dq[:1000], few, torch.cuda.current_stream())
        if mapped:
            want_h = want.cpu()
            hq, ho = q.pin_memory(), torch.empty((nq, 3)).pin_memory()
            del dq, want
            torch.cuda.empty_cache()
        else:
            got = torch.empty_like(want)
        torch.cuda.synchronize()
        try:
            # all but less than the call's buffers (64 MB for the sort alone)
            while (free := torch.cuda.mem_get_info()[0]) > 48 << 20:
                part = max((free - (24 << 20)) & ~((2 << 20) - 1), 2 << 20)
                while part >= 2 << 20:
                    try:
                        fill.append(torch.empty(part, dtype=torch.uint8, device="cuda"))
                        break
                    except torch.OutOfMemoryError:
                        part //= 2
                else:
                    break
            assert torch.cuda.mem_get_info()[0] < 60 << 20
            if mapped:
                c2.check(c2.lib.pm_photonmap_radiance(
                    c2.handle, 0, hq.data_ptr(), nq, K, N, ho.data_ptr()),
                    "pm_photonmap_radiance")
            else:
                call(c2, dq, got, torch.cuda.current_stream())
                torch.cuda.synchronize()
        finally:
            fill.clear()
            torch.cuda.empty_cache()
        if mapped:
            np.testing.assert_array_equal(ho.numpy(), want_h.numpy())
        else:
            assert torch.equal(got, want)


def test_calls_on_one_stream_share_a_buffer(own):
    """Eight calls in flight on one stream, then calls that grow by 2 % each: the
    memory taken is that of one buffer, enlarged once."""
    import torch
    nq = 2_000_000
    q = torch.from_numpy(W.wall_queries(nq + nq // 3, 5)).cuda()
    out = torch.empty((q.shape[0], 3), device="cuda")
    st = torch.cuda.Stream()
    call(own, q[:1000], out, st)  # kernels loaded
    call(own, q[:MIN_QUERIES], out, st)
    torch.cuda.synchronize()
    free = [torch.cuda.mem_get_info()[0]]
    for _ in range(8):
        call(own, q[:nq], out, st)
    torch.cuda.synchronize()
    free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[1] < 2 * 17 * nq  # 16 bytes per query and the sort's table
    for i in range(15):
        call(own, q[:nq + nq // 50 * i], out, st)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert len(set(free[1:])) <= 2
    torch.cuda.synchronize()


def test_call_beside_a_capture(own):
    """A call on a stream that captures nothing, while another stream's capture (in
    the global mode, the default) goes on."""
    import torch
    q = torch.from_numpy(W.wall_queries(MIN_QUERIES, 6)).cuda()
    with Context(0) as c2:
        pm = PhotonMap(c2)
        pm.setPhotons(W.wall_photons(N, 1))
        pm.build()
        want = alone(c2, q)  # kernels loaded
    x, got = torch.zeros(1, device="cuda"), torch.empty_like(want)
    other, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        x.add_(1)
        call(own, q, got, other)
        x.add_(1)
    g.replay()
    torch.cuda.synchronize()
    assert x.item() == 2
    assert torch.equal(got, want)
    del g
