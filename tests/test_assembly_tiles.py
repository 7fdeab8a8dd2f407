"""Assembly at the edges of the element-pair kernel's tiles, on a B200.

The kernel integrates unordered pairs of square tiles (32 faces in FP32, 16 in
FP64).  Face counts here lie one below, at and above one and several tiles,
with and without the x symmetry's image pass.  The FP64 system matches the
oracle's within 1e-12 of the largest entry (36 to 1,536 terms of round-off per
entry), the FP32 one within 2e-6 (the FP32 phase), as in the parity tests.
"""
import numpy as np
import pytest

import oracle
from beat_engine_b200 import _lib
from beat_engine_b200 import mesh as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("faces", [15, 16, 17, 31, 32, 33, 48, 65, 96])
@pytest.mark.parametrize("mode", ["off", "x"])
def test_system_entries(faces, mode):
    whole = M.uv_sphere_patch(0.1, 7, 8, -np.pi / 2, np.pi / 2)  # 96 faces
    f = whole.faces[:faces]
    used = np.unique(f)
    index = np.full(whole.num_vertices, -1)
    index[used] = np.arange(used.size)
    mesh = M.BoundaryMesh(whole.vertices[used], index[f], np.ones(faces, dtype=np.int32))
    k = -11.0
    rng = np.random.default_rng(faces)
    q = rng.standard_normal((faces, 3)) + 1j * rng.standard_normal((faces, 3))
    Ao, bo = (oracle.assemble(mesh, k, 1.0 / k, q) if mode == "off" else
              oracle.assemble_sym(mesh, k, 1.0 / k, q, mode))
    with _lib.Context(0) as c:
        c.set_symmetry(mode)
        c.set_mesh(mesh.vertices, mesh.faces, 4, 4)
        for prec, tol in ((_lib.FP64, 1e-12), (_lib.MIXED_FP32_IR, 2e-6)):
            A, b = c.assemble(k, 1.0 / k, q, prec)
            assert np.max(np.abs(A - Ao)) <= tol * np.max(np.abs(Ao)), (prec, "A")
            assert np.max(np.abs(b - bo)) <= tol * np.max(np.abs(bo)), (prec, "b")
            # one column alone takes the matrix-free right-hand side
            A, b = c.assemble(k, 1.0 / k, q[:, :1], prec)
            assert np.max(np.abs(b - bo[:, :1])) <= tol * np.max(np.abs(bo[:, :1])), (prec, "b, matrix-free")
