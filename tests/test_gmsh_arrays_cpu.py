"""The array parser of Gmsh 2.2 sections against the loop over lines (meshes.py).

Every form the loop accepts either gives the same mesh from the array parser or is left to
the loop (None): other element types between the triangles, node ids out of order and not
dense, references to unknown nodes, tags, scales, irregular spacing, signs, repeated ids.
"""

import numpy as np
import pytest

from conftest import pkg_module

meshes = pkg_module("meshes")

NODES = ["1 0 0 0", "2 1e-1 0 0", "4 0 0.25 -1.5E-3", "3 0.1 0.2 0.30000000000000004"]
ELEMS = ["1 2 2 7 1 1 2 4", "2 2 2 3 1 4 2 3"]


def same(a, b):
    return (np.array_equal(a.vertices, b.vertices) and np.array_equal(a.faces, b.faces)
            and np.array_equal(a.tags, b.tags) and a.faces.dtype == b.faces.dtype and a.tags.dtype == b.tags.dtype)


@pytest.mark.parametrize("nodes,elems,arrays", [
    (NODES, ELEMS, True),
    (NODES, ["9 15 2 1 1 3", *ELEMS, "10 1 2 5 1 1 2"], True),          # points and lines between
    (NODES, [*ELEMS, "3 2 2 3 1 4 2 99"], True),                        # unknown node: dropped
    (NODES, [*ELEMS, "4 2 3 8 1 0 1 3 2"], True),                       # three tags
    ([n.replace(" ", "  ") for n in NODES], ELEMS, False),              # double spaces
    (NODES, [e.replace(" ", "\t") for e in ELEMS], False),              # tabs
    ([*NODES, "2 0.5 0.5 0.5"], ELEMS, False),                          # repeated id
    ([*NODES, "1000000 0.5 0.5 0.5"], ELEMS, False),                    # sparse ids
    (NODES, ["1 2 2 -7 1 1 2 4"], False),                               # a signed tag
    ([*NODES, "5 1 2"], ELEMS, False),                                  # a short line
    ([*NODES, "5 1 2 3 4"], ELEMS, False),                              # a long one
])
@pytest.mark.parametrize("scale", [1.0, 0.001])
def test_array_parser_agrees_with_the_loop(nodes, elems, arrays, scale):
    got = meshes._gmsh22_arrays(nodes, elems, scale)
    assert (got is not None) == arrays
    if got is not None:
        assert same(got, meshes._gmsh22_lines(nodes, elems, scale))


def test_written_meshes_round_trip(tmp_path):
    box = meshes.box_with_piston((0.3, 0.2, 0.25), 700, 0.05, "+z")
    path = tmp_path / "box.msh"
    meshes.write_gmsh22(path, box.vertices, box.faces, box.tags)
    got = meshes.read_gmsh22(path)
    assert np.array_equal(got.vertices, box.vertices) and np.array_equal(got.faces, box.faces)
    assert np.array_equal(got.tags, box.tags)
