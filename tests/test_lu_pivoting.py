"""The LU where rows do move, on a B200.

The Burton-Miller systems of the other tests keep their pivots on or near the
diagonal, so a factorisation that loses an interchange can pass them.  A
strong random admittance makes A + B diag(a) P far from diagonally dominant:
most columns then pivot to a distant row.  Sizes lie on both sides of a
sub-panel's width (32 columns in FP32, 16 in FP64), of a panel's (128) and of
the rows of one CTA (256), with last sub-panels of two columns and up.

Bounds, derived from the systems: both forms solve the operator they
assembled, so against a dense FP64 solution the FP64 form's error is its
round-off times the condition number (checked below 1e6: 1e-9), the mixed
form's the FP32 assembly's 1e-7 times it (1e-1 at most, with the refinement's
residual at its 1e-10 target against its own operator).
"""
import numpy as np
import pytest

import oracle
from beat_engine_b200 import _lib
from beat_engine_b200 import mesh as M
from oracle import adjoint as adj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("faces", [60, 100, 250, 290, 520, 1050])
def test_solution_with_distant_pivots(faces):
    mesh = M.rounded_box_enclosure(faces, seed=faces)
    k, n = 18.0, mesh.num_vertices
    rng = np.random.default_rng(faces)
    A, B = adj.operators(mesh, k, 1.0 / k)
    P = adj.face_average(mesh)
    a = 200.0 * (rng.standard_normal(mesh.num_faces) + 1j * rng.standard_normal(mesh.num_faces))
    S = A + B @ (a[:, None] * P)
    cond = np.linalg.cond(S)
    assert cond < 1e6
    assert np.mean(np.argmax(np.abs(S.real) + np.abs(S.imag), axis=0) != np.arange(n)) > 0.25
    q = rng.standard_normal((mesh.num_faces, 2)) + 1j * rng.standard_normal((mesh.num_faces, 2))
    ref = np.linalg.solve(S, B @ q)
    with _lib.Context(0) as c:
        c.set_mesh(mesh.vertices, mesh.faces, 4, 4)
        c.set_admittance(a)
        for nb in (32, 64, 128, 256):
            p, d = c.solve(k, 1.0 / k, q, _lib.Context.opts(_lib.FP64, lu_block=nb))
            assert np.linalg.norm(p - ref) <= 1e-14 * cond * np.linalg.norm(ref), (n, nb)
            p, d = c.solve(k, 1.0 / k, q, _lib.Context.opts(_lib.MIXED_FP32_IR, lu_block=nb))
            assert d["precision"] == _lib.MIXED_FP32_IR and d["ir_converged"] == 1 and d["ir_iterations"] <= 8, (n, nb, d)
            assert np.linalg.norm(p - ref) <= 1e-6 * cond * np.linalg.norm(ref), (n, nb)
