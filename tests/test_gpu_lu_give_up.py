"""The LU panels' bounded waits: an exchange that gives up ends the call with an error, writes
nothing outside the matrix, and leaves the context usable.

With a limit of no reads every CTA gives up at the first column; with a few, some CTAs may
have their words and others not, at any column.  Whatever happens the factorisation either
returns the usual factors or the error, and the next one, with the default limit, is the
same to the bit as before.
"""

import numpy as np
import pytest

from conftest import pkg_module

pytestmark = pytest.mark.gpu
meshes = pkg_module("meshes")
native = pkg_module("native")

MIXED, FP64 = native.BEM_PRECISION_MIXED, native.BEM_PRECISION_FP64


@pytest.mark.parametrize("precision,n", [(MIXED, 700), (MIXED, 2600), (FP64, 96), (FP64, 700), (FP64, 2600)])
@pytest.mark.parametrize("reads", [0, 1, 3])
def test_dense_factorisation(precision, n, reads):
    rng = np.random.default_rng(n)
    a = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    ctx = native.Context(0)
    try:
        lu, ipiv = ctx.lu_factor_dense(a, precision=precision)
        ctx.set_exchange_limit(reads)
        try:
            lu1, ipiv1 = ctx.lu_factor_dense(a, precision=precision)
            assert reads > 0 and np.array_equal(lu1, lu) and np.array_equal(ipiv1, ipiv)
        except native.BemError as exc:
            assert "gave up waiting" in str(exc)
        ctx.set_exchange_limit()
        lu2, ipiv2 = ctx.lu_factor_dense(a, precision=precision)
        assert np.array_equal(lu2, lu) and np.array_equal(ipiv2, ipiv)
    finally:
        ctx.close()


@pytest.mark.parametrize("precision,n_freq,lanes", [(MIXED, 2, 1), (MIXED, 8, 2), (FP64, 3, 1)])
def test_solve(precision, n_freq, lanes):
    v, f = meshes.cube_sphere(0.1, 11)  # 728 vertices: a cluster of two CTAs in the mixed form
    freqs = np.geomspace(300.0, 1500.0, n_freq)
    ctx = native.Context(0)
    try:
        m = ctx.upload_mesh(v, f)
        m.set_excitation((v[f].mean(axis=1)[:, 2] > 0.08).astype(np.complex128)[None, :])
        m.set_observation_points(np.array([[0, 0, 2.0], [0, 1.2, 1.6]]))
        p, u, _ = m.solve(freqs, precision=precision, lanes=lanes)
        ctx.set_exchange_limit(0)
        with pytest.raises(native.BemError, match="gave up waiting"):
            m.solve(freqs, precision=precision, lanes=lanes)
        ctx.set_exchange_limit()
        p2, u2, _ = m.solve(freqs, precision=precision, lanes=lanes)
        assert np.array_equal(p2, p) and np.array_equal(u2, u)
    finally:
        ctx.close()
