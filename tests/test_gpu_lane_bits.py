"""Two lanes give the bits of one stream, also where a call's one batch is dealt to both.

What could tell the lanes' halves from the whole batch: the last outer block's width and the
residual's column splits (orders around 1,000 and 2,500 lie where they depend on the batch),
the field's split of the faces (by points and frequencies), the geometry that frequencies
share in fours and twos, and a refinement step that only one half needs.
"""

import numpy as np
import pytest

from conftest import pkg_module

pytestmark = pytest.mark.gpu
native = pkg_module("native")
meshes = pkg_module("meshes")
request = pkg_module("request")


def _check(gpu_ctx, mesh, drives, points, freqs, precision, batches, **kw):
    m = gpu_ctx.upload_mesh(mesh.vertices, mesh.faces, symmetry=kw.pop("symmetry", "off"))
    try:
        m.set_excitation(drives)
        m.set_observation_points(points)
        p1, u1, s1 = m.solve(freqs, precision=precision, **kw)
        p2, u2, s2 = m.solve(freqs, precision=precision, lanes=2, **kw)
    finally:
        m.release()
    assert s1["batches"] == 1 and s2["batches"] == batches
    assert np.array_equal(p1, p2) and np.array_equal(u1, u2)


@pytest.mark.parametrize("faces,n_rhs", [(300, 1), (1100, 1), (2000, 2), (2000, 4), (5000, 1)])
@pytest.mark.parametrize("n_freq", [8, 12, 13, 16])
def test_mixed(gpu_ctx, faces, n_rhs, n_freq):
    mesh = meshes.box_with_piston((0.4, 0.3, 0.35), faces, 0.08, "+z")
    d = (mesh.tags == meshes.RADIATOR_TAG).astype(np.complex128)
    drives = np.stack([d * np.exp(0.7j * i) for i in range(n_rhs)])
    _check(gpu_ctx, mesh, drives, request.fibonacci_sphere(700, 2.0), np.geomspace(200.0, 2000.0, n_freq),
           native.BEM_PRECISION_MIXED, 2)


@pytest.mark.parametrize("n_freq,batches", [(8, 2), (11, 1), (16, 2)])
def test_fp64(gpu_ctx, n_freq, batches):
    mesh = meshes.box_with_piston((0.4, 0.3, 0.35), 600, 0.08, "+z")
    d = (mesh.tags == meshes.RADIATOR_TAG).astype(np.complex128)
    _check(gpu_ctx, mesh, np.stack([d, 1j * d]), request.fibonacci_sphere(300, 2.0),
           np.geomspace(200.0, 2000.0, n_freq), native.BEM_PRECISION_FP64, batches)


def test_symmetric_mesh(gpu_ctx):
    half = meshes.fundamental_domain(meshes.box_with_piston((0.4, 0.3, 0.35), 3000, 0.08, "+z"), "x")
    d = (half.tags == meshes.RADIATOR_TAG).astype(np.complex128)
    _check(gpu_ctx, half, np.stack([d, 1j * d]), request.fibonacci_sphere(300, 2.0),
           np.geomspace(200.0, 2000.0, 12), native.BEM_PRECISION_MIXED, 2, symmetry="x")


def test_a_step_that_one_half_needs(gpu_ctx):
    """A tolerance between the residuals of two frequencies: the first half is done one step
    before the second, and its frequencies stay where they would be without the other half."""
    mesh = meshes.box_with_piston((0.4, 0.3, 0.35), 600, 0.08, "+z")
    d = (mesh.tags == meshes.RADIATOR_TAG).astype(np.complex128)[None, :]
    freqs = np.geomspace(200.0, 2000.0, 8)
    m = gpu_ctx.upload_mesh(mesh.vertices, mesh.faces)
    try:
        m.set_excitation(d)
        m.set_observation_points(request.fibonacci_sphere(64, 2.0))
        kw = dict(precision=native.BEM_PRECISION_MIXED, refine_tol=1.0)  # accepts the first solution
        first = [m.solve(freqs[i:i + 4], batch=4, **kw)[2]["max_rel_residual"] for i in (0, 4)]
        assert first[0] != first[1]
        kw["refine_tol"] = float(np.sqrt(first[0] * first[1]))
        p1, u1, s1 = m.solve(freqs, **kw)
        p2, u2, s2 = m.solve(freqs, lanes=2, **kw)
    finally:
        m.release()
    assert s1["batches"] == 1 and s2["batches"] == 2 and s1["max_refine_steps"] == 1
    assert np.array_equal(p1, p2) and np.array_equal(u1, u2)
