"""The mixed form's LU at the edges of its outer blocks: the last block takes up to 1,024
columns of one matrix, the ones before 256 each, and the last panel may be partial.

Backward error ||P A - L U|| / ||A||: where all updates are IEEE FP32 (up to 1,024) that of
LAPACK's complex64 factorisation of the same matrix, with half as much again for another
order of the sums; 1e-4 where tensor-core updates take part.
"""

import numpy as np
import pytest
import scipy.linalg

from conftest import pkg_module

pytestmark = pytest.mark.gpu
native = pkg_module("native")


def backward_error(a, lu, ipiv):
    n = len(a)
    perm = np.arange(n)
    for i, p in enumerate(ipiv):
        perm[[i, p]] = perm[[p, i]]
    lu = lu.astype(np.complex128)
    L, U = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    return np.linalg.norm(a[perm] - L @ U) / np.linalg.norm(a), L


@pytest.mark.parametrize("n", [31, 33, 256, 257, 288, 512, 513, 1023, 1024, 1025, 1281])
def test_backward_error(gpu_ctx, n):
    rng = np.random.default_rng(n)
    a = (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))) / np.sqrt(n)
    lu, ipiv = gpu_ctx.lu_factor_dense(a, precision=native.BEM_PRECISION_MIXED)
    err, L = backward_error(a, lu, ipiv)
    assert np.abs(L).max() <= np.sqrt(2.0) * (1.0 + 1e-5)
    ref, _ = backward_error(a, *scipy.linalg.lu_factor(a.astype(np.complex64)))
    assert err < (1.5 * ref if n <= 1024 else 1e-4), (err, ref)


@pytest.mark.parametrize("edge,n_freq", [(9, 1), (9, 7), (10, 2), (13, 1), (13, 4)])
def test_batches_reach_the_refinement(gpu_ctx, edge, n_freq):
    """Orders 488, 602 and 1,016, where the batch decides how wide the last block is."""
    v, f = pkg_module("meshes").cube_sphere(0.1, edge)
    m = gpu_ctx.upload_mesh(v, f)
    try:
        m.set_excitation((v[f].mean(axis=1)[:, 2] > 0.08).astype(np.complex128)[None, :])
        m.set_observation_points(np.array([[0, 0, 2.0], [0, 1.2, 1.6]]))
        freqs = np.geomspace(200.0, 1800.0, n_freq)
        p, _, st = m.solve(freqs, precision=native.BEM_PRECISION_MIXED)
        q = np.concatenate([m.solve([fr], precision=native.BEM_PRECISION_MIXED)[0] for fr in freqs])
    finally:
        m.release()
    assert st["max_rel_residual"] <= 1e-10 and st["max_refine_steps"] <= 2
    assert np.all(np.linalg.norm(p - q, axis=(1, 2)) <= 1e-8 * np.linalg.norm(q, axis=(1, 2)))
