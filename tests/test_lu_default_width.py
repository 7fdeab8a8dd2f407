"""The default panel width of a single solve, on a B200: 32 columns up to 3,072
unknowns, 128 above and in sweeps, on both sides of the line.

Bounds: the two widths factor the same operator.  In FP64 they differ by its
round-off times a condition number below 1e4 (1e-10); in the mixed form each
solves its own FP32 assembly, whose sums differ in the last bits by the order
of their additions, to a residual of 1e-10 (1e-6).
"""
import numpy as np
import pytest

from beat_engine_b200 import _lib
from beat_engine_b200 import mesh as M

pytestmark = pytest.mark.gpu


def mesh_of(vertices):
    """A rounded box with exactly that many vertices: faces split at their centroids."""
    box = M.rounded_box_enclosure(6140 if vertices > 1000 else 60, seed=1)
    X, F = box.vertices.copy(), box.faces.copy()
    for i in range(vertices - box.num_vertices):
        a, b, c = F[i]
        X = np.vstack([X, X[[a, b, c]].mean(axis=0)])
        v = len(X) - 1
        F = np.vstack([F, [[b, c, v], [c, a, v]]])
        F[i] = (a, b, v)
    return M.BoundaryMesh(X, F.astype(box.faces.dtype), np.ones(len(F), dtype=np.int32))


@pytest.mark.parametrize("vertices,width", [(34, 32), (3072, 32), (3073, 128)])
@pytest.mark.parametrize("precision,tol", [(_lib.FP64, 1e-10), (_lib.MIXED_FP32_IR, 1e-6)])
def test_default_width_of_a_single_solve(vertices, width, precision, tol):
    mesh = mesh_of(vertices)
    assert mesh.num_vertices == vertices
    k = 9.0
    rng = np.random.default_rng(vertices)
    q = rng.standard_normal((mesh.num_faces, 2)) + 1j * rng.standard_normal((mesh.num_faces, 2))
    with _lib.Context(0) as c:
        c.set_mesh(mesh.vertices, mesh.faces, 4, 4)
        p, d = c.solve(k, 1.0 / k, q, _lib.Context.opts(precision))
        p2, d2 = c.solve(k, 1.0 / k, q, _lib.Context.opts(precision, lu_block=160 - width))
    assert (d["lu_block"], d2["lu_block"]) == (width, 160 - width)
    assert d["precision"] == precision and d["ir_converged"] == 1
    assert np.linalg.norm(p - p2) <= tol * np.linalg.norm(p2)
