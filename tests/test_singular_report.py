"""What a solve of an exactly singular system reports, on a B200.

A vertex that no face uses has a row and a column of zeros, so its pivot is an
exact zero: at the first column or at the last.  The status of a factorisation
is read with the first wait of its solve, after the substitutions have been
queued; every form of the solve has to raise BEAT_B200_SINGULAR all the same,
leave no factors behind, and leave the context usable.
"""
import numpy as np
import pytest

from beat_engine_b200 import _lib
from beat_engine_b200 import mesh as M

pytestmark = pytest.mark.gpu
K = 30.0


@pytest.mark.parametrize("place", ["first", "last"])
@pytest.mark.parametrize("level", [1, 2])  # 43 and 163 unknowns: one panel and two
def test_unused_vertex(place, level):
    import torch

    m = M.reference_sphere(0.1, level)
    verts, tri = np.asarray(m.vertices), np.asarray(m.faces)
    extra = np.array([[0.0, 0.0, 0.5]])
    bad = (np.concatenate([extra, verts]), tri + 1) if place == "first" else (np.concatenate([verts, extra]), tri)
    rng = np.random.default_rng(level)
    q = rng.standard_normal((m.num_faces, 2)) + 1j * rng.standard_normal((m.num_faces, 2))
    forms = [(_lib.FP64, 0), (_lib.MIXED_FP32_IR, 0), (_lib.MIXED_FP32_IR, _lib.FLAG_NO_REFINE)]
    with _lib.Context(0) as c:
        for prec, flags in forms:
            c.set_mesh(bad[0], bad[1], 4, 4)
            n = bad[0].shape[0]
            x = torch.zeros(n, dtype=torch.complex128, device="cuda")
            for _ in range(3):  # eager, then as the factorisation's graph
                with pytest.raises(_lib.BeatB200Error) as e:
                    c.solve(K, 1.0 / K, q, _lib.Context.opts(prec, flags=flags))
                assert e.value.status == _lib.SINGULAR, (prec, flags)
                with pytest.raises(_lib.BeatB200Error) as e:
                    c.resolve_noalloc(1, x.data_ptr(), x.data_ptr())
                assert e.value.status == _lib.STATE
            c.set_mesh(verts, tri, 4, 4)
            p, d = c.solve(K, 1.0 / K, q, _lib.Context.opts(prec, flags=flags))
            A, b = c.assemble(K, 1.0 / K, q, _lib.FP64)
            assert np.linalg.norm(p - np.linalg.solve(A, b)) <= 1e-5 * np.linalg.norm(p)
