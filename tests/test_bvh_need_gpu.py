"""The traversal stack's limits (csrc/pm_scene.cuh) on trees that need them: what a
stack setting accepts is what the walk of the binary tree fits in.

Scenes as in test_bvh_stack_gpu.py: equal boxes, so that the tree over n faces is
balanced, with ceil(log2(n)) levels, and a ray inside the boxes pushes a node on every
level but the last: 131,072 faces need 16 entries, one face more 17."""
from __future__ import annotations

import numpy as np
import pytest

from photon_mapping_b200 import _native as N
from photon_mapping_b200 import batch as B
from photon_mapping_b200 import scene as S
from photon_mapping_b200.camera import Camera
from test_bvh_stack_gpu import N_CHAIN_BITS, N_LIGHTS, deep_chain_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("faces,fits", [(4096, True), (65536, True), (65537, True),
                                        (131072, True), (160016, False)])
def test_sixteen_entries(faces, fits):
    cam = Camera(S.CAMERA["position"], S.CAMERA["forward"], S.CAMERA["fov"])
    mesh = deep_chain_mesh(faces - 2 * N_CHAIN_BITS - N_LIGHTS)
    assert mesh.n_faces == faces
    br = B.BatchRenderer([dict(mesh=mesh, camera=cam, width=8, height=8, spp=1, k=10,
                               photons=200, seed=5, max_depth=4)])
    try:
        br.set_tuning(bvh_stack=64)
        br.render(use_graph=False)
        img, ph = br.image(0), br.photons(0)
        br.set_tuning(bvh_stack=16)
        if not fits:
            with pytest.raises(N.PMError) as e:
                br.render(use_graph=False)
            assert e.value.status == N.PM_ERR_DEVICE_STATUS
            return
        br.render(use_graph=False)
        np.testing.assert_array_equal(br.image(0), img)
        np.testing.assert_array_equal(br.photons(0), ph)
    finally:
        br.close()
