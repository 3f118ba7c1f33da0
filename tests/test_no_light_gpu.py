"""Final gathering in a scene without emitting faces, on photons that the caller set:
there is no light to sample, so direct light is zero and the image is the gathered
estimates alone."""
from __future__ import annotations

import numpy as np
import pytest

from photon_mapping_b200 import scene as S
from photon_mapping_b200 import workloads as W
from photon_mapping_b200.camera import Camera
from photon_mapping_b200.integrator import PhotonMapping

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", (S.cornell_box(0), S.caustics_scene(0, grid=10, subdiv=1)),
                         ids=("lambert", "specular"))
def test_gathering_without_lights(ctx, mesh):
    mesh = S.Mesh(**{**vars(mesh), "materials": np.array(mesh.materials, copy=True)})
    mesh.materials["le"] = 0.0
    sc = S.Scene(ctx)
    sc.setMesh(mesh)
    sc.build()
    cam = Camera(S.CAMERA["position"], S.CAMERA["forward"], S.CAMERA["fov"])
    pmi = PhotonMapping(1000, 20, 1.0, 20, 1, 20, ctx=ctx)
    pmi.global_map.setPhotons(W.wall_photons(20000, 1))
    pmi.global_map.build()
    pmi.caustics_map.setPhotons(np.zeros((0, 9), np.float32))
    pmi.caustics_map.build()
    for m in (0, 1):
        ctx.check(ctx.lib.pm_photonmap_set_emitted(ctx.handle, m, 20000), "pm_photonmap_set_emitted")
    img, st = pmi.render(cam, 40, 30, 2, n_gather=3)
    assert np.isfinite(img).all() and (img >= 0).all() and img.max() > 0
    assert st["dropped_nan"] == 0 and st["queries_caustics"] > 0
