"""Which FP64 calls go through the Chebyshev moments: those of at least 12 frequencies of which
enough converge to pay for the terms, by the call's own frequencies only.

On the sphere of 1,280 triangles (edges of 1.4 cm) frequencies up to 4 kHz need 12 to 16 terms
and none above 40 kHz converges, so of 12 frequencies one does not pay and ten do.
"""

import numpy as np
import pytest

from conftest import pkg_module

pytestmark = pytest.mark.gpu
native = pkg_module("native")
meshes = pkg_module("meshes")


@pytest.mark.parametrize("low,through", [(1, 0), (2, 0), (10, 10), (12, 12)])
def test_calls_through_the_moments(gpu_ctx, low, through):
    mesh = meshes.sphere_with_cap(0.1, 3, 30.0)
    freqs = np.concatenate([np.linspace(800.0, 1000.0, low), np.linspace(40000.0, 45000.0, 12 - low)])
    m = gpu_ctx.upload_mesh(mesh.vertices, mesh.faces)
    try:
        m.set_excitation((mesh.tags == meshes.RADIATOR_TAG).astype(np.complex128)[None, :])
        m.set_observation_points(np.array([[0.0, 0.0, 2.0]]))
        for _ in range(2):  # the second time after a call that formed the moments
            st = m.solve(freqs, precision=native.BEM_PRECISION_FP64)[2]
            assert st["singular_cheb_freqs"] == through
            m.solve(np.linspace(700.0, 1000.0, 12), precision=native.BEM_PRECISION_FP64)
    finally:
        m.release()
