"""CudaEngine.device_bytes against the scratch that the solve then holds, on the lanes it uses.

The estimate also has the mesh's own data and slack, so it is at least the scratch; the
extended rows of the second lane are what a split call adds.
"""

import numpy as np
import pytest

from conftest import pkg_module

pytestmark = pytest.mark.gpu
native = pkg_module("native")
meshes = pkg_module("meshes")
engine = pkg_module("engine")


@pytest.mark.parametrize("precision,faces,n_freq,lanes,batch,n_rhs,batches",
                         [("mixed", 600, 8, 2, 0, 1, 2), ("mixed", 2500, 11, 2, 0, 2, 1), ("mixed", 2500, 12, 2, 0, 4, 2),
                          ("mixed", 10000, 15, 1, 0, 1, 1), ("mixed", 10000, 15, 2, 0, 1, 2),
                          ("mixed", 10000, 9, 2, 6, 1, 2), ("fp64", 1300, 16, 2, 0, 1, 2), ("fp64", 5000, 8, 2, 0, 1, 2)])
def test_estimate_covers_the_scratch(precision, faces, n_freq, lanes, batch, n_rhs, batches):
    mesh = meshes.box_with_piston((0.4, 0.3, 0.35), faces, 0.08, "+z")
    drive = (mesh.tags == meshes.RADIATOR_TAG).astype(np.complex128)
    e = engine.CudaEngine(precision=precision, context="thread", lanes=lanes, batch=batch)
    e.ctx = native.Context(0)  # nothing held from other tests
    try:
        e.prepare(mesh.vertices, mesh.faces, np.stack([drive] * n_rhs), np.random.default_rng(0).normal(size=(2000, 3)) * 3)
        estimate = e.device_bytes(n_freq)
        stats = e.solve(np.geomspace(200.0, 2000.0, n_freq), 343.0, 1.205).stats
        assert stats["batches"] == batches
        assert estimate >= e.ctx.scratch_bytes, (estimate, e.ctx.scratch_bytes)
    finally:
        ctx = e.ctx
        e.close()
        ctx.close()
