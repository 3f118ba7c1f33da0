"""Batches whose estimates are answered by tiles of sorted queries (csrc/pm_knn_tile.cu,
knn_tile_batch_kernel): images bit-identical to the per-scene loop."""
from __future__ import annotations

import numpy as np
import pytest

from photon_mapping_b200 import batch as B
from photon_mapping_b200 import scene as S
from photon_mapping_b200.camera import Camera

pytestmark = pytest.mark.gpu


def box_scene(k, photons, seed, side=160, spp=2, **kw):
    cam = Camera(S.CAMERA["position"], S.CAMERA["forward"], S.CAMERA["fov"])
    return dict(dict(mesh=S.cornell_box(0), camera=cam, width=side, height=side, spp=spp, k=k,
                     photons=photons, seed=seed, max_depth=20), **kw)


def check(scenes, min_work, tuned=()):
    seq = B.Sequential(scenes)
    want, _ = seq.render()
    seq.close()
    br = B.BatchRenderer(scenes)
    try:
        stored, queries = br.counts()
        # work by which tiles are chosen: queries x (largest k + 50)
        assert queries.sum() * (max(s["k"] for s in scenes) + 50) >= min_work
        for t in ({},) + tuple(tuned):
            br.set_tuning(**t)
            for use_graph in (False, True):
                br.render(use_graph=use_graph)
                for i, w in enumerate(want):
                    np.testing.assert_array_equal(br.image(i), w)
        return stored, queries
    finally:
        br.close()


@pytest.mark.parametrize("ks", [(50, 20, 100, 50, 1), (300, 50, 448, 20, 7)])
def test_tiled_batch(ks):
    """Full maps of several k, a scene without photons, scenes with maps too small for
    tiles and ragged query counts."""
    scenes = [box_scene(ks[0], 40000, 1), box_scene(ks[1], 0, 2, side=33),
              box_scene(ks[2], 30000, 3, side=97, spp=3), box_scene(ks[3], 700, 4, side=61),
              box_scene(ks[4], 20, 5, side=45)]
    stored, _ = check(scenes, 2 * 2_500_000, tuned=(dict(knn_warps=4, knn_buffer=2048),))
    assert stored[1] == 0 and 20 < stored[3] < 4096 and 0 < stored[4] < 4096
    assert min(stored[0], stored[2]) >= 4096


@pytest.mark.parametrize("photons", (0, 900))
def test_batch_of_small_maps_only(photons):
    """Queries enough for tiles, and no map that takes them."""
    stored, _ = check([box_scene(50, photons, s, side=128) for s in range(4)], 2 * 2_500_000,
                      tuned=(dict(knn_chunk=7),))
    assert max(stored) < 4096


def test_autotune_of_a_tiled_batch_leaves_the_chunk_alone():
    """Tiles have work items of their own: nothing to measure knn_chunk by."""
    br = B.BatchRenderer([box_scene(50, 20000, 6)])
    try:
        br.render()
        img = br.image(0)
        br.set_tuning(knn_chunk=24)
        best, _ = br.autotune()
        assert best["knn_chunk"] == 24
        br.render()
        np.testing.assert_array_equal(br.image(0), img)
    finally:
        br.close()
