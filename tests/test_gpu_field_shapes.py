"""The FP32 field kernel over the shapes its dispatch knows: rules of one, three and six
points (an odd rule's last point stands alone), one to four excitations, groups of one, two
and four frequencies with a partly filled last group, point counts around a warp, and faces
with and without a normal velocity.  Against the CPU oracle at the mixed form's 1e-5.
"""

import numpy as np
import pytest

from conftest import pkg_module

pytestmark = pytest.mark.gpu
meshes = pkg_module("meshes")
C, RHO = 343.0, 1.205


@pytest.mark.parametrize("order,nrhs,n_freq,n_points", [
    (1, 1, 1, 1), (1, 1, 5, 33), (2, 1, 1, 31), (2, 1, 7, 200), (2, 3, 2, 32), (4, 1, 1, 65),
    (4, 1, 3, 31), (4, 1, 6, 33), (4, 2, 3, 100), (4, 3, 2, 1), (4, 4, 2, 40), (1, 4, 3, 64)])
def test_field_matches_oracle(gpu_ctx, native, order, nrhs, n_freq, n_points):
    from oracle import oracle

    mesh = meshes.box_with_piston((0.3, 0.2, 0.25), 220, 0.08, "+z")
    rng = np.random.default_rng(10 * order + nrhs)
    piston = (mesh.tags == meshes.RADIATOR_TAG)
    drives = (rng.normal(size=(nrhs, mesh.n_faces)) + 1j * rng.normal(size=(nrhs, mesh.n_faces))) * piston
    pts = rng.normal(size=(n_points, 3))
    pts *= (0.6 + rng.random(size=(n_points, 1))) / np.linalg.norm(pts, axis=1, keepdims=True)
    freqs = np.linspace(250.0, 1100.0, n_freq)
    m = gpu_ctx.upload_mesh(mesh.vertices, mesh.faces, order)
    try:
        m.set_excitation(drives)
        m.set_observation_points(pts)
        _, u, _ = m.solve(freqs, precision=native.BEM_PRECISION_MIXED, sound_speed=C, rho=RHO)
    finally:
        m.release()
    for i in sorted({0, n_freq // 2, n_freq - 1}):
        omega = 2 * np.pi * freqs[i]
        ref = oracle.solve_frequency(mesh, omega / C, (drives * 1j * RHO * omega).T, pts, regular_order=order)
        for c in range(nrhs):
            assert np.linalg.norm(u[i, c] - ref.field[:, c]) / np.linalg.norm(ref.field[:, c]) < 1e-5


@pytest.mark.parametrize("order,nrhs,n_freq", [(1, 1, 1), (2, 1, 2), (4, 1, 3), (4, 1, 4), (4, 1, 5), (2, 1, 8), (4, 2, 3),
                                               (1, 2, 2), (4, 3, 2), (4, 4, 1)])
def test_fp64_field_of_a_call_equals_single_frequencies(gpu_ctx, native, order, nrhs, n_freq):
    """The FP64 field kernel's groups of one, two and four frequencies: each frequency by
    itself, so a call of several agrees with single ones to the 1e-12 of their pressures (FP64
    rounding times a condition below 1e3)."""
    mesh = meshes.box_with_piston((0.3, 0.2, 0.25), 160, 0.08, "+z")
    rng = np.random.default_rng(order + 7 * nrhs)
    drives = rng.normal(size=(nrhs, mesh.n_faces)) * (mesh.tags == meshes.RADIATOR_TAG)
    pts = rng.normal(size=(37, 3))
    pts *= 1.2 / np.linalg.norm(pts, axis=1, keepdims=True)
    freqs = np.linspace(250.0, 1100.0, n_freq)
    m = gpu_ctx.upload_mesh(mesh.vertices, mesh.faces, order)
    try:
        m.set_excitation(drives.astype(np.complex128))
        m.set_observation_points(pts)
        _, u, _ = m.solve(freqs, precision=native.BEM_PRECISION_FP64, sound_speed=C, rho=RHO)
        one = [m.solve([f], precision=native.BEM_PRECISION_FP64, sound_speed=C, rho=RHO)[1][0] for f in freqs]
    finally:
        m.release()
    for i in range(n_freq):
        assert np.linalg.norm(u[i] - one[i]) <= 1e-12 * np.linalg.norm(one[i])
