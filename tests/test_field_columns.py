"""Field and far field for every pass width of the evaluator, on a B200: one
and two right-hand sides in registers, then products of 4, 8 and 16, alone and
after a full pass of 16, with point counts around the 32 of a CTA and source
counts that are no multiple of a chunk.  FP64 sums of F Q terms against the
oracle: 1e-11 of each column's norm, as in the parity tests.
"""
import numpy as np
import pytest

import oracle
from beat_engine_b200 import _lib
from beat_engine_b200 import mesh as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns", [1, 2, 3, 4, 5, 8, 9, 16, 17, 18, 19, 23, 29])
@pytest.mark.parametrize("points", [1, 31, 33, 70])
def test_columns(columns, points):
    mesh = M.rounded_box_enclosure(90, seed=columns)
    k = 25.0
    rng = np.random.default_rng(100 * columns + points)

    def z(n):
        return rng.standard_normal((n, columns)) + 1j * rng.standard_normal((n, columns))

    p, q = z(mesh.num_vertices), z(mesh.num_faces)
    x = M.fibonacci_sphere(points, 0.6)
    with _lib.Context(0) as c:
        c.set_mesh(mesh.vertices, mesh.faces, 4, 4)
        for got, ref in ((c.field(k, x, p, q), oracle.field(mesh, k, x, p, q)),
                         (c.farfield(k, x, p, q), oracle.farfield(mesh, k, x, p, q))):
            err = np.linalg.norm(got - ref, axis=0) / np.linalg.norm(ref, axis=0)
            assert np.all(err <= 1e-11), err
