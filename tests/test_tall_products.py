"""The products of the stored operators with a few columns, on a B200: B q of
the assembly, A x inside the refinement, and their conjugate transposes in the
adjoint, at column counts on both sides of a block of 8 and of a pass of 16,
with face counts (row strides, reduction lengths) that are no multiple of
anything.

Bounds: those of the parity and adjoint tests; b is a sum of at most 300
products in FP64 (1e-12 of its largest entry), FP32 entries of B give 2e-6;
gradients 1e-9 and 2e-6 in relative L2.
"""
import numpy as np
import pytest

from beat_engine_b200 import _lib
from beat_engine_b200 import mesh as M
from oracle import adjoint as adj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("faces", [17, 63, 287])
def test_products_with_few_columns(faces):
    whole = M.uv_sphere_patch(0.1, 13, 13, -np.pi / 2, np.pi / 2)
    f = whole.faces[:faces]
    assert len(f) == faces
    used = np.unique(f)
    index = np.full(whole.num_vertices, -1)
    index[used] = np.arange(used.size)
    mesh = M.BoundaryMesh(whole.vertices[used], index[f], np.ones(faces, dtype=np.int32))
    k = 11.0
    A, B = adj.operators(mesh, k, 1.0 / k)
    P = adj.face_average(mesh)
    dirs = M.fibonacci_sphere(7, 1.0)
    Fp, Fq = adj.farfield_operators(mesh, k, dirs)
    rng = np.random.default_rng(faces)
    zero = np.zeros(faces, dtype=np.complex128)
    with _lib.Context(0) as c:
        c.set_mesh(mesh.vertices, mesh.faces, 4, 4)
        for R in (1, 2, 8, 9, 16, 17, 33):
            q = rng.standard_normal((faces, R)) + 1j * rng.standard_normal((faces, R))
            g = rng.standard_normal((7, R)) + 1j * rng.standard_normal((7, R))
            b, p = B @ q, np.linalg.solve(A, B @ q)
            w, ga = adj.adjoint(A, B, P, zero, Fp, Fq, p, g)
            for prec, tol, gtol in ((_lib.FP64, 1e-12, 1e-9), (_lib.MIXED_FP32_IR, 2e-6, 2e-6)):
                _, bd = c.assemble(k, 1.0 / k, q, prec, want_matrix=False)
                assert np.max(np.abs(bd - b)) <= tol * np.max(np.abs(b)), (R, prec, "b")
                pd, d = c.solve(k, 1.0 / k, q, _lib.Context.opts(prec, flags=_lib.FLAG_RHS_CACHED))
                assert d["precision"] == prec and d["ir_converged"] == 1
                assert np.linalg.norm(pd - p) <= gtol * np.linalg.norm(p), (R, prec, "p")
                wd, _ = c.adjoint(k, dirs, pd, g, _lib.Context.opts(prec), want_admittance=False)
                assert np.linalg.norm(wd - w) <= gtol * np.linalg.norm(w), (R, prec, "w")
