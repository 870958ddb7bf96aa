"""Calls of one automatic batch on two lanes: split in two where both halves have four
frequencies, with the results of one lane.

A frequency's system does not depend on which others share its launches, so the traces
agree to the refinement's 1e-10 (tolerance 1e-9) in the mixed form and to rounding times
the condition (1e-12) in the FP64 form.
"""

import numpy as np
import pytest

from conftest import pkg_module

pytestmark = pytest.mark.gpu
meshes = pkg_module("meshes")


@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (1, 1e-9)])
@pytest.mark.parametrize("n_freq,batches", [(1, 1), (7, 1), (8, 2), (9, 1), (11, 1), (12, 2), (13, 2), (16, 2)])
def test_split_call_matches_one_lane(gpu_ctx, n_freq, batches, precision, tol):
    mesh = meshes.box_with_piston((0.3, 0.2, 0.25), 300, 0.06, "+z")
    freqs = np.geomspace(200.0, 3000.0, n_freq)
    m = gpu_ctx.upload_mesh(mesh.vertices, mesh.faces)
    try:
        m.set_excitation((mesh.tags == meshes.RADIATOR_TAG).astype(np.complex128)[None, :])
        m.set_observation_points(np.array([[0.0, 0.0, 2.0], [1.5, 0.3, 1.2]]))
        p1, u1, s1 = m.solve(freqs, precision=precision)
        p2, u2, s2 = m.solve(freqs, precision=precision, lanes=2)
    finally:
        m.release()
    assert s1["batches"] == 1 and s2["batches"] == batches
    assert s1["singular_cheb_freqs"] == s2["singular_cheb_freqs"]
    for a, b in ((p2, p1), (u2, u1)):
        assert np.all(np.linalg.norm(a - b, axis=(1, 2)) <= tol * np.linalg.norm(b, axis=(1, 2)))
