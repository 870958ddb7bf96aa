"""Calls on a device with next to no memory left: what ran without the second lane's scratch or
the FP64 form's moments still runs without them, with the same results.

The context has solved the same mesh before (its scratch and kernels are there), then the
rest of the device's memory is taken.
"""

import contextlib

import numpy as np
import pytest

from conftest import pkg_module

pytestmark = pytest.mark.gpu
native = pkg_module("native")
meshes = pkg_module("meshes")


@contextlib.contextmanager
def device_full():
    """Holds the device's free memory but for a few tens of MB."""
    import torch

    held = []
    for size in (1 << 32, 1 << 28, 1 << 25):
        while True:
            try:
                held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                break
    try:
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def _upload(ctx, faces):
    mesh = meshes.box_with_piston((0.4, 0.3, 0.35), faces, 0.08, "+z")
    m = ctx.upload_mesh(mesh.vertices, mesh.faces)
    m.set_excitation((mesh.tags == meshes.RADIATOR_TAG).astype(np.complex128)[None, :])
    m.set_observation_points(np.array([[0.0, 0.0, 2.0], [1.5, 0.3, 1.2]]))
    return m


def test_fp64_sweep_without_room_for_moments():
    """About 4 KB a pair: 200 MB for 4,000 triangles, which a call of 12 frequencies would hold."""
    freqs = np.geomspace(200.0, 900.0, 12)
    kw = dict(precision=native.BEM_PRECISION_FP64, batch=1)
    ctx = native.Context(0)
    try:
        m = _upload(ctx, 4000)
        p, u, st = m.solve(freqs[:11], **kw)
        assert st["singular_cheb_freqs"] == 0
        with device_full():
            p1, u1, st = m.solve(freqs, **kw)
        assert st["singular_cheb_freqs"] == 0
        assert np.array_equal(p1[:11], p) and np.array_equal(u1[:11], u)
        _, _, st = m.solve(freqs, **kw)  # with memory again
        assert st["singular_cheb_freqs"] == 12
    finally:
        ctx.close()


def test_split_call_without_room_for_the_second_lane():
    freqs = np.geomspace(200.0, 1500.0, 8)
    kw = dict(precision=native.BEM_PRECISION_MIXED)
    ctx = native.Context(0)
    try:
        m = _upload(ctx, 5000)
        p, u, st = m.solve(freqs, **kw)
        assert st["batches"] == 1
        with device_full():
            p1, u1, st = m.solve(freqs, lanes=2, **kw)
        assert st["batches"] == 1
        assert np.array_equal(p1, p) and np.array_equal(u1, u)
        p2, u2, st = m.solve(freqs, lanes=2, **kw)  # with memory again
        assert st["batches"] == 2
        assert np.array_equal(p2, p) and np.array_equal(u2, u)
    finally:
        ctx.close()


def test_an_allocation_that_failed_is_reported_once():
    ctx = native.Context(0)
    try:
        m = _upload(ctx, 5000)
        with device_full(), pytest.raises(native.BemError, match="OUT_OF_MEMORY"):
            m.solve([700.0])
        assert m.solve([700.0])[2]["max_rel_residual"] <= 1e-10
        _upload(ctx, 600).release()
    finally:
        ctx.close()
