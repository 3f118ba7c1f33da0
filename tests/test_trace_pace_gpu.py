"""The two paces of the photon trace (csrc/pm_trace.cu, trace_pace): with few
photons a warp's lanes shade together, with many they shade as they finish.

A photon's path depends on its index and the seed alone, so the photons that the
first indices of a large trace store are those of a small trace (which the
oracle tests cover), bit for bit, in the same order.
"""
from __future__ import annotations

import numpy as np
import pytest

from photon_mapping_b200 import PhotonMap
from photon_mapping_b200 import scene as S
from photon_mapping_b200.integrator import trace_photons

pytestmark = pytest.mark.gpu

FULL = 4 * 148 * 24 * 32  # photons from which the lanes run apart (148 SMs)


@pytest.mark.parametrize("scene", ["box", "specular"])
@pytest.mark.parametrize("map_id", [0, 1])
def test_many_photons_begin_like_few(ctx, scene, map_id):
    mesh = S.cornell_box(0) if scene == "box" else S.caustics_scene(0, grid=24, subdiv=2)
    sc = S.Scene(ctx)
    sc.setMesh(mesh)
    sc.build()
    pm = PhotonMap(ctx, map_id)
    few = trace_photons(ctx, map_id, 11, 20_000, 100)
    want = pm.photons()
    many = trace_photons(ctx, map_id, 11, FULL + 12_345, 100)
    got = pm.photons()
    assert many["emitted"] == FULL + 12_345 and got.shape[0] == many["stored"]
    assert few["stored"] == want.shape[0]
    assert (scene == "box" and map_id == 1) == (few["stored"] == 0)
    np.testing.assert_array_equal(got[:want.shape[0]], want)
