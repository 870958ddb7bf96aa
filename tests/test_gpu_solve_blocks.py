"""Solves through the inverted diagonal blocks (mixed form) at orders around the block edges.

Cube spheres of 6 n^2 + 2 vertices give orders below one 32-row block (26), of one and two
256-row outer blocks with a ragged last one (218, 296), and of several (488, 728), with one
to four right-hand sides in a cluster's shared reads.  Pressure and field against the FP64
CPU oracle at the mixed form's bound (1e-5); the refinement must reach its 1e-10 in at most
two steps, as it does with substituted blocks.
"""

import numpy as np
import pytest

from conftest import pkg_module

pytestmark = pytest.mark.gpu
meshes = pkg_module("meshes")
C, RHO = 343.0, 1.205


@pytest.mark.parametrize("n,nrhs", [(2, 1), (6, 2), (7, 3), (9, 4), (11, 1)])
def test_block_solves_match_oracle(gpu_ctx, native, n, nrhs):
    from oracle import oracle

    v, f = meshes.cube_sphere(0.1, n)
    mesh = meshes.BoundaryMesh(v, f, np.ones(len(f), np.int32))
    rng = np.random.default_rng(n)
    drives = rng.normal(size=(nrhs, len(f))) + 1j * rng.normal(size=(nrhs, len(f)))
    pts = np.array([[0, 0, 2.0], [2.0, 0, 0], [0, 1.2, 1.6]])
    freqs = [300.0, 900.0]
    m = gpu_ctx.upload_mesh(v, f)
    try:
        m.set_excitation(drives)
        m.set_observation_points(pts)
        p, u, st = m.solve(freqs, precision=native.BEM_PRECISION_MIXED, sound_speed=C, rho=RHO)
    finally:
        m.release()
    assert st["max_rel_residual"] <= 1e-10 and st["max_refine_steps"] <= 2
    for i, fr in enumerate(freqs):
        omega = 2 * np.pi * fr
        ref = oracle.solve_frequency(mesh, omega / C, (drives * 1j * RHO * omega).T, pts)
        for c in range(nrhs):
            assert np.linalg.norm(p[i, c] - ref.pressure[:, c]) / np.linalg.norm(ref.pressure[:, c]) < 1e-5
            assert np.linalg.norm(u[i, c] - ref.field[:, c]) / np.linalg.norm(ref.field[:, c]) < 1e-5
