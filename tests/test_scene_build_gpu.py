"""The tree build in one cooperative launch (csrc/pm_scene.cu, ploc_kernel) at
the sizes where it changes: the largest cluster count that one block takes alone
(4,096), the first that several blocks share, and counts that leave blocks with
uneven or empty shares. Closest hits equal the oracle's brute force bit for bit
on a context whose scene is replaced again and again.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from photon_mapping_b200 import scene as S

pytestmark = pytest.mark.gpu


def mesh_of(n_faces, seed):
    """n_faces random small triangles, a light among them."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, 1, (n_faces, 1, 3))
    tris = (c + rng.normal(size=(n_faces, 3, 3)) * 0.05).reshape(n_faces, 9)
    m = S.mesh_from_triangles(tris[1:], S.material(rho=S.WHITE), "white") if n_faces > 1 else None
    light = S.mesh_from_triangles(tris[:1], S.material(le=(1.0, 1.0, 1.0)), "light")
    return light if m is None else light + m


@pytest.mark.parametrize("n_faces", [4096, 4097, 1, 2, 3, 4099, 37_889, 5_000, 257])
def test_hits_equal_brute_force(ctx, n_faces):
    mesh = mesh_of(n_faces, n_faces)
    sc = S.Scene(ctx)
    sc.setMesh(mesh)
    sc.build()
    rng = np.random.default_rng(1)
    o = rng.uniform(-0.5, 1.5, (600, 3)).astype(np.float32)
    d = rng.normal(size=(600, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    d[:30, rng.integers(0, 3, 30)] = 0.0  # axis-parallel directions among them
    got = sc.intersect(o, d)
    r = np.empty((o.shape[0], 8), np.float32)
    r[:, 0:3], r[:, 3], r[:, 4:7], r[:, 7] = o, 1e-5, d, np.finfo(np.float32).max
    want = O.OracleScene(mesh).intersect(r)
    np.testing.assert_array_equal(got["prim"], want[:, 3].view(np.int32))
    hit = got["prim"] >= 0
    for i, name in enumerate("tuv"):
        np.testing.assert_array_equal(got[name][hit], want[hit, i])
