"""The camera pass of scenes with only Lambert surfaces (rays of one sample in
their own threads, csrc/pm_render.cu) against the path-per-thread pass: the same
scene with a speck of mirror that no ray meets takes that one. Every sample draws
the same random numbers, so the images, ray counts and sampler states are equal."""
from __future__ import annotations

import numpy as np
import pytest

from photon_mapping_b200 import scene as S
from photon_mapping_b200.camera import Camera
from photon_mapping_b200.integrator import PhotonMapping

pytestmark = pytest.mark.gpu


def speck():
    """A mirror of 1e-4 behind the left wall, a box length away from the room."""
    p = np.array([[[-1.0, 0.5, 0.5], [-1.0, 0.5001, 0.5], [-1.0, 0.5, 0.5001]]])
    m = S.mesh_from_triangles(p, S.material(rho=(0.9, 0.9, 0.9)), "speck")
    m.materials["type"] = 1
    return m


def pair(ctx, n_photons, k, fg, max_depth, seed):
    for mesh in (S.cornell_box(2), S.cornell_box(2) + speck()):
        scene = S.Scene(ctx)
        scene.setMesh(mesh)
        scene.build()
        pmi = PhotonMapping(n_photons, k, 1.0, k, fg, max_depth, ctx=ctx)
        pmi.build(scene, seed=seed)
        yield pmi


@pytest.mark.parametrize("fg", (0, 1))
@pytest.mark.parametrize("w,h,spp,n_gather,batch,max_depth,back",
                         [(33, 17, 5, 1, 0, 100, 0.0), (16, 16, 3, 7, 2, 100, 1.5), (1, 1, 4, 64, 1, 1, 0.0),
                          (40, 9, 1, 2, 0, 2, 4.0)])
def test_split_pass_is_the_path_pass(ctx, w, h, spp, n_gather, batch, max_depth, back, fg):
    pos = np.asarray(S.CAMERA["position"], np.float32) - back * np.asarray(S.CAMERA["forward"],
                                                                           np.float32)
    cam = Camera(pos, S.CAMERA["forward"], S.CAMERA["fov"])
    got = [pmi.render(cam, w, h, spp, n_gather=n_gather, spp_batch=batch)
           for pmi in pair(ctx, 5000, 20, fg, max_depth, 3)]
    assert np.isfinite(got[0][0]).all()
    np.testing.assert_array_equal(got[0][0], got[1][0])
    for key in ("rays", "queries_global", "queries_caustics", "dropped_nan", "dropped_negative"):
        assert got[0][1][key] == got[1][1][key], key


@pytest.mark.parametrize("fg", (0, 1))
def test_integrated_rays_and_their_samplers(ctx, fg):
    rng = np.random.default_rng(1)
    n = 129
    o = rng.uniform(0.1, 0.9, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    st = rng.integers(0, 1 << 62, n).astype(np.uint64)
    got = [pmi.integrate_batch(o, d, st, n_gather=3) for pmi in pair(ctx, 5000, 20, fg, 100, 3)]
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])


def test_estimates_in_an_empty_map_are_zero(ctx):
    """Lambert scenes store no caustics photons: their caustics estimates are
    zeros written without a search, which statistics switch on again."""
    cam = Camera(S.CAMERA["position"], S.CAMERA["forward"], S.CAMERA["fov"])
    scene = S.Scene(ctx)
    scene.setMesh(S.cornell_box(2))
    scene.build()
    pmi = PhotonMapping(5000, 20, 1.0, 20, 1, 100, ctx=ctx)
    pmi.build(scene, seed=3)
    img, st = pmi.render(cam, 31, 17, 2)
    assert st["queries_caustics"] > 0
    ctx.set_stats(True)
    try:
        want, wst = pmi.render(cam, 31, 17, 2)
    finally:
        ctx.set_stats(False)
    np.testing.assert_array_equal(img, want)
    assert st["queries_caustics"] == wst["queries_caustics"]
