"""The FP64 form's LU at the edges of its panels: 32 columns, one row to a thread of at most
16 x 256, the 64-wide panel beyond, and the partial panel at the end.

Pivots identical to LAPACK's and factors within 1e-11, as for the other orders; a column
of zeros is reported; solves with either panel width agree to 1e-12 (condition below 1e3).
"""

import numpy as np
import pytest
import scipy.linalg

from conftest import pkg_module

pytestmark = pytest.mark.gpu
meshes = pkg_module("meshes")


@pytest.mark.parametrize("n", [31, 32, 33, 63, 96, 257, 1025, 4096, 4097])
def test_pivots_and_factors(gpu_ctx, native, n):
    rng = np.random.default_rng(n)
    a = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    lu, ipiv = gpu_ctx.lu_factor_dense(a, precision=native.BEM_PRECISION_FP64)
    lu_ref, piv_ref = scipy.linalg.lu_factor(a)
    assert np.array_equal(ipiv, piv_ref)
    assert np.linalg.norm(lu - lu_ref) / np.linalg.norm(lu_ref) < 1e-11


def test_equal_candidates_take_the_first_row_and_low_words_decide(gpu_ctx, native):
    n = 96
    rng = np.random.default_rng(5)
    a = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    a[:, 0] = 1.0                       # all rows tie: row 0
    a[:, 1] = a[0, 1] + 1.0             # after the first step all rows tie again: row 1
    a[40, 1] += 2.0 ** -50              # but one, in the last bits
    _, ipiv = gpu_ctx.lu_factor_dense(a, precision=native.BEM_PRECISION_FP64)
    _, piv_ref = scipy.linalg.lu_factor(a)
    assert ipiv[0] == 0 and np.array_equal(ipiv, piv_ref)


@pytest.mark.parametrize("col", [0, 31, 32, 95])
def test_zero_column_is_reported(gpu_ctx, native, col):
    a = np.random.default_rng(col).normal(size=(96, 96)).astype(np.complex128)
    a[:, col] = 0.0
    with pytest.raises(native.BemError, match="SINGULAR"):
        gpu_ctx.lu_factor_dense(a, precision=native.BEM_PRECISION_FP64)


@pytest.mark.parametrize("edge,n_freq", [(5, 1), (8, 5), (8, 24), (13, 3)])
def test_panel_widths_agree_in_solves(gpu_ctx, native, edge, n_freq):
    v, f = meshes.cube_sphere(0.1, edge)  # 6 edge^2 + 2 vertices
    m = gpu_ctx.upload_mesh(v, f)
    try:
        m.set_excitation((v[f].mean(axis=1)[:, 2] > 0.08).astype(np.complex128)[None, :])
        m.set_observation_points(np.array([[0, 0, 2.0], [0, 1.2, 1.6]]))
        freqs = np.geomspace(200.0, 1800.0, n_freq)
        p = [m.solve(freqs, precision=native.BEM_PRECISION_FP64, lu_block=w)[0] for w in (0, 32, 64)]
    finally:
        m.release()
    for q in p[1:]:
        assert np.all(np.linalg.norm(q - p[0], axis=(1, 2)) <= 1e-12 * np.linalg.norm(p[0], axis=(1, 2)))
