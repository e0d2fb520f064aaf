"""Mesh volume maps skip groups of 32 faces: face counts at and beside a group's size, faces in
an order that scatters each group over the whole surface, and the oracle's map of the same mesh,
with the bounds of test_gpu_mesh.py (signs wherever |phi| > 1e-3; the reference's quadratic form
cancels 4e-7 C of the squared distance, C the squared extent of the map)."""
import numpy as np
import pytest

import vfd_gb300 as V
from oracle import oracle as O
from vfd_gb300 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("segments,shuffled", [(3, False), (16, True), (17, False), (65, True)])
def test_groups_of_faces(segments, shuffled):
    v, t = meshes.cone((0, 0, 0), 0.3, 0.5, segments)
    if shuffled:
        t = t[np.random.default_rng(segments).permutation(len(t))]
    a = V.build_mesh_map(v, t, None, False, 0.0, (9, 11, 7), 0.02)
    b = O.build_mesh_map(v, t, None, False, 0.0, (9, 11, 7), 0.02)
    np.testing.assert_array_equal(a.cells, b.cells)
    nn, m = a.struct.node_count, a.meta()
    da, db = a.nodes[:nn].astype(np.float64), b.nodes[:nn].astype(np.float64)
    far = np.abs(db) > 1e-3
    assert np.all(np.sign(da[far]) == np.sign(db[far]))
    C = float(np.sum((np.asarray(m["domain_max"]) - np.asarray(m["domain_min"])) ** 2))
    assert np.all(np.abs(da - db) <= 2e-6 + 4e-7 * C / np.maximum(np.abs(db), np.sqrt(4e-7 * C)))
