"""The LU's panel kernel at every number of rows per thread, with rows that
move far, on a B200.

A thread of the panel kernel holds one row (up to 2,048 rows left), two (on 128
threads up to 4,096, on 256 up to 8,192) or three; one CTA alone takes the last
128.  A factorisation passes through all of them from its size downwards.  A
strong random admittance on a mesh with shuffled vertex numbers makes A + B
diag(a) P pivot far from the diagonal, so that each variant has to exchange
rows of its own threads, of other threads and of other CTAs.

The operators come from the device (the coupled export), the system and its
residual are formed by torch.  Bounds on |S p - B q| / (|S| |p|), Frobenius
norms: FP64, N u (partial pivoting with an element growth far above what
occurs); mixed, 1e-6, five times its FP32 operators' rounding.  Its refinement
gains at least a factor of ten per iteration while the condition number times
2^-24 is below 0.1 (1e4 at 2,370 unknowns), so 12 reach 1e-10 with room.
"""
import numpy as np
import pytest

from beat_engine_b200 import _lib
from beat_engine_b200 import mesh as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("faces, more_than", [(4300, 2048), (8500, 4096), (16800, 8192)])
def test_residual_with_distant_pivots(faces, more_than):
    import torch

    whole = M.rounded_box_enclosure(faces, seed=faces)
    rng = np.random.default_rng(faces)
    order = rng.permutation(whole.num_vertices)
    number = np.argsort(order).astype(np.int32)
    verts, tri = np.asarray(whole.vertices)[order], number[np.asarray(whole.faces)]
    N, F, R, k = whole.num_vertices, whole.num_faces, 2, 18.0
    assert more_than < N <= more_than * 1.1
    a = 2000.0 * (rng.standard_normal(F) + 1j * rng.standard_normal(F))
    q = rng.standard_normal((F, R)) + 1j * rng.standard_normal((F, R))
    z = {"dtype": torch.complex128, "device": "cuda"}
    S, C = torch.zeros(N, N, **z), torch.zeros(F, N, **z)  # columns first: S[j, i], C[f, i]
    torch.cuda.synchronize()
    with _lib.Context(0) as c:
        c.set_mesh(verts, tri, 4, 4)
        c.assemble_coupled_device(k, _lib.FP64, S.data_ptr(), C.data_ptr())  # C = -B
        b = torch.from_numpy(q).cuda().T @ -C
        at = torch.from_numpy(tri.astype(np.int64)).cuda()
        D = (torch.from_numpy(a).cuda() / 3.0)[:, None] * C
        for v in range(3):
            S.index_add_(0, at[:, v], D, alpha=-1)
        pivots = (S.real.abs() + S.imag.abs()).argmax(dim=1)
        assert ((pivots - torch.arange(N, device="cuda")).abs() > 64).double().mean() > 0.25
        c.set_admittance(a)
        for prec, bound in ((_lib.FP64, N * 2.0 ** -53), (_lib.MIXED_FP32_IR, 1e-6)):
            p, d = c.solve(k, 1.0 / k, q, _lib.Context.opts(prec))
            assert d["precision"] == prec
            if prec != _lib.FP64:
                assert d["ir_converged"] == 1 and d["ir_iterations"] <= 12, d
            x = torch.from_numpy(np.ascontiguousarray(p.T)).cuda()
            assert (x @ S - b).norm() <= bound * S.norm() * x.norm(), (N, prec)
