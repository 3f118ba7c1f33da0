"""Contexts and batches that are alive together and use different k or launch shapes:
the kernels' shared-memory limits belong to the process, so none may set one that
another's launch exceeds."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from photon_mapping_b200 import Context, PhotonMap
from photon_mapping_b200 import batch as B
from photon_mapping_b200 import scene as S
from photon_mapping_b200 import workloads as W
from photon_mapping_b200.camera import Camera

pytestmark = pytest.mark.gpu


def box_scene(k, seed):
    """About 45,000 estimates: tiles answer them from k = 6 on."""
    cam = Camera(S.CAMERA["position"], S.CAMERA["forward"], S.CAMERA["fov"])
    return dict(mesh=S.cornell_box(0), camera=cam, width=160, height=160, spp=2, k=k,
                photons=20000, seed=seed, max_depth=20)


def sequential(scenes):
    seq = B.Sequential(scenes)
    try:
        return seq.render()[0]
    finally:
        seq.close()


def test_two_batches_of_different_k():
    sets = [[box_scene(300, 1)], [box_scene(50, 2)]]
    want = [sequential(s) for s in sets]
    brs = [B.BatchRenderer(s) for s in sets]
    try:
        for br in brs:
            _, queries = br.counts()
            assert queries.sum() * (50 + 50) >= 2_500_000  # tiles
        for use_graph in (False, True):
            for br, w in zip(brs, want):
                br.render(use_graph=use_graph)
                np.testing.assert_array_equal(br.image(0), w[0])
        brs[0].set_tuning(block=64)  # drops the graph: captured again
        brs[0].render(use_graph=True)
        np.testing.assert_array_equal(brs[0].image(0), want[0][0])
    finally:
        for br in brs:
            br.close()


def test_two_batches_of_different_warps():
    """Few queries: the warp-per-query kernel with the tuning's shape."""
    scenes = [dict(box_scene(20, 3), width=24, height=24, photons=2000)]
    want = sequential(scenes)
    brs = [B.BatchRenderer(scenes) for _ in range(2)]
    try:
        brs[0].set_tuning(knn_warps=8, knn_buffer=2048)
        brs[1].set_tuning(knn_warps=1, knn_buffer=2048)
        for use_graph in (False, True):
            for br in brs:
                br.render(use_graph=use_graph)
                np.testing.assert_array_equal(br.image(0), want[0])
    finally:
        for br in brs:
            br.close()


def test_two_contexts_of_different_k_in_two_threads():
    ph = W.wall_photons(20000, 1)
    errors = []

    def work(k):
        try:
            q = W.wall_queries(5_000_000 // (k + 50) + 1, k)
            with Context(0) as ctx:
                pm = PhotonMap(ctx)
                pm.setPhotons(ph)
                pm.build()
                want = pm.radiance(q, k, 20000)
                for _ in range(60):
                    if not np.array_equal(pm.radiance(q, k, 20000), want):
                        errors.append(f"k={k}: another result")
                        return
        except Exception as e:  # noqa: BLE001
            errors.append(f"k={k}: {e}")

    threads = [threading.Thread(target=work, args=(k,)) for k in (448, 200)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
