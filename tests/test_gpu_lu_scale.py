"""Dense LU of matrices scaled by a power of two: the same pivots and multipliers to the bit and
the scaled U, also where the pivots' squares leave the exponent range (2^-126 .. 2^128 in
FP32, 2^-1022 .. 2^1024 in FP64).

Orders on both sides of one CTA's rows in the panels; every update is IEEE FP32 or FP64, so
nothing but the pivot's inverse sees the scale.
"""

import numpy as np
import pytest

from conftest import pkg_module

pytestmark = pytest.mark.gpu
native = pkg_module("native")


@pytest.mark.parametrize("precision,n,exps", [(native.BEM_PRECISION_MIXED, 100, (-70, -50, 50, 70)),
                                              (native.BEM_PRECISION_MIXED, 700, (-70, -50, 50, 70)),
                                              (native.BEM_PRECISION_FP64, 96, (-520, -450, 450, 520)),
                                              (native.BEM_PRECISION_FP64, 700, (-520, -450, 450, 520))])
def test_scaled_matrix(gpu_ctx, precision, n, exps):
    rng = np.random.default_rng(n)
    a = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    lu, ipiv = gpu_ctx.lu_factor_dense(a, precision=precision)
    for e in exps:
        lu_s, ipiv_s = gpu_ctx.lu_factor_dense(a * 2.0**e, precision=precision)
        assert np.array_equal(ipiv_s, ipiv), e
        assert np.array_equal(np.tril(lu_s, -1), np.tril(lu, -1)), e
        assert np.array_equal(np.triu(lu_s), np.triu(lu) * 2.0**e), e
