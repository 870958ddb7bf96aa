"""FP64 sweeps: what a call shares between its frequencies does not change any of them.

A call of at least 12 frequencies integrates the singular remainder through the mesh's
Chebyshev moments, a shorter one point by point; the regular pairs take two frequencies
per block and all frequencies of a batch in one launch.  Tolerance: the moments are cut at
5e-16 and everything else is FP64, so the sums differ by a few 1e-16 of the rows' scale;
the condition of these systems is below 1e3, which leaves 1e-12.  One sweep is also held
against the CPU oracle at the FP64 form's 1e-9.
"""

import numpy as np
import pytest

from conftest import pkg_module

pytestmark = pytest.mark.gpu
meshes = pkg_module("meshes")
C, RHO = 343.0, 1.205
PTS = np.array([[0, 0, 2.0], [2.0, 0, 0], [0, 1.2, 1.6]])


def upload(gpu_ctx, mesh):
    m = gpu_ctx.upload_mesh(mesh.vertices, mesh.faces)
    m.set_excitation((mesh.tags == meshes.RADIATOR_TAG).astype(np.complex128)[None, :])
    m.set_observation_points(PTS)
    return m


def close(a, b):
    return np.all(np.linalg.norm(a - b, axis=(1, 2)) <= 1e-12 * np.linalg.norm(b, axis=(1, 2)))


@pytest.mark.parametrize("faces,f_hi,beyond", [(200, 2500.0, 0), (450, 900.0, 0), (200, 12000.0, 1)])
def test_long_sweep_equals_short_ones_and_oracle(gpu_ctx, native, faces, f_hi, beyond):
    from oracle import oracle

    mesh = meshes.box_with_piston((0.3, 0.2, 0.25), faces, 0.06, "+z")
    freqs = np.concatenate([np.geomspace(40.0, min(f_hi, 2500.0), 12), [f_hi]])
    m = upload(gpu_ctx, mesh)
    try:
        p, u, st = m.solve(freqs, precision=native.BEM_PRECISION_FP64, sound_speed=C, rho=RHO)
        assert 6 <= st["singular_cheb_freqs"] <= len(freqs) - beyond
        parts = [m.solve(fs, precision=native.BEM_PRECISION_FP64, sound_speed=C, rho=RHO)
                 for fs in (freqs[:6], freqs[6:])]
        assert all(s["singular_cheb_freqs"] == 0 for _, _, s in parts)
    finally:
        m.release()
    assert close(p, np.concatenate([q[0] for q in parts]))
    assert close(u, np.concatenate([q[1] for q in parts]))
    i = 7
    omega = 2 * np.pi * freqs[i]
    drive = (mesh.tags == meshes.RADIATOR_TAG).astype(np.complex128)
    ref = oracle.solve_frequency(mesh, omega / C, drive * 1j * RHO * omega, PTS)
    assert np.linalg.norm(p[i, 0] - ref.pressure[:, 0]) / np.linalg.norm(ref.pressure[:, 0]) < 1e-9
    assert np.linalg.norm(u[i, 0] - ref.field[:, 0]) / np.linalg.norm(ref.field[:, 0]) < 1e-9


@pytest.mark.parametrize("n_freq,batch", [(2, 0), (3, 0), (5, 2), (11, 0), (40, 0), (16, 3)])
def test_frequencies_of_a_call_equal_single_ones(gpu_ctx, native, n_freq, batch):
    mesh = meshes.box_with_piston((0.3, 0.2, 0.25), 150, 0.06, "+z")
    freqs = np.geomspace(100.0, 2000.0, n_freq)
    m = upload(gpu_ctx, mesh)
    try:
        p, u, _ = m.solve(freqs, precision=native.BEM_PRECISION_FP64, sound_speed=C, rho=RHO, batch=batch)
        for i in range(0, n_freq, max(1, n_freq // 5)):
            pi, ui, _ = m.solve(freqs[i:i + 1], precision=native.BEM_PRECISION_FP64, sound_speed=C, rho=RHO)
            assert close(p[i:i + 1], pi) and close(u[i:i + 1], ui), i
    finally:
        m.release()
