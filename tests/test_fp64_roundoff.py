"""Round-off of the FP64 form on a B200.

u = 2^-53.  A stage that sums small terms apart before it adds them to what is
large, and whose rounding errors have no common sign, stays within a few u of
its exact result at these sizes; the bounds below are that, not the parity
tests' 1e-11, which would hide the loss of three digits.
"""
import numpy as np
import pytest

import oracle
from beat_engine_b200 import _lib
from beat_engine_b200 import mesh as M

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _complex(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _distance(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("mode, bound", [("off", 10), ("x", 30)])
def test_right_hand_side(mode, bound):
    """Most of a right-hand side's entry comes from the touching pairs of its
    own faces.  Twice the oracle's own error, which in long double arithmetic is
    5 u here and 16 u with the image's pairs."""
    mesh = M.reference_sphere(0.1, 2) if mode == "off" else M.uv_sphere_patch(0.1, 12, 12, -np.pi / 2, np.pi / 2)
    k = 20.0
    q = _complex(np.random.default_rng(1), mesh.num_faces, 1)
    _, bo = (oracle.assemble(mesh, k, 1.0 / k, q) if mode == "off" else
             oracle.assemble_sym(mesh, k, 1.0 / k, q, mode))
    with _lib.Context(0) as c:
        c.set_symmetry(mode)
        c.set_mesh(mesh.vertices, mesh.faces, 4, 4)
        _, b = c.assemble(k, 1.0 / k, q, _lib.FP64, want_matrix=False)
    assert _distance(b, bo) <= bound * U


def _refined(A, b):
    """A^-1 b to well below u: residuals in long double, corrections in FP64."""
    Al, bl = A.astype(np.clongdouble), b.astype(np.clongdouble)
    inverse = np.linalg.inv(A)
    x = (inverse @ b).astype(np.clongdouble)
    for _ in range(3):
        r = np.stack([bl[:, c] - (Al * x[:, c]).sum(axis=1) for c in range(b.shape[1])], axis=1)
        x += inverse @ r.astype(np.complex128)
    return x


@pytest.mark.parametrize("faces, lu_block", [(600, 128), (1992, 128), (1992, 32), (1992, 256)])
def test_solution(faces, lu_block):
    """The factorisation's products are small against the entries they change, so
    what counts is how often an entry is rounded at its own magnitude: once per
    step of its sub-panel (16), once per sub-panel of its panel and once per
    panel, 30 to 50 times here, with random signs and u / 2 to u / 3 each time,
    and about as much again in the substitutions: 8 u.  (Rounded there twice per
    index, 2,000 times, the error was 18 u at 998 unknowns.)"""
    mesh = M.rounded_box_enclosure(faces, seed=faces)
    k = 20.0
    q = _complex(np.random.default_rng(2), mesh.num_faces, 2)
    with _lib.Context(0) as c:
        c.set_mesh(mesh.vertices, mesh.faces, 4, 4)
        p, _ = c.solve(k, 1.0 / k, q, _lib.Context.opts(_lib.FP64, flags=_lib.FLAG_RHS_CACHED, lu_block=lu_block))
        A, b = c.assemble(k, 1.0 / k, q, _lib.FP64)
    assert _distance(p, _refined(A, b)) <= 8 * U


@pytest.mark.parametrize("faces", [100, 300])
@pytest.mark.parametrize("columns", [2, 9, 16])
def test_mapping_times_columns(faces, columns):
    """b = B q against the long double product with the device's own B (its
    product with the identity is exact).  A chain of n terms of random signs,
    then K / n such sums, have an error of sqrt(n + K / 2n) roundings in rms, of
    u / sqrt(3) at most each; n = 16."""
    mesh = M.rounded_box_enclosure(faces, seed=faces)
    k, n = 20.0, mesh.num_faces
    q = _complex(np.random.default_rng(columns), n, columns)
    with _lib.Context(0) as c:
        c.set_mesh(mesh.vertices, mesh.faces, 4, 4)
        _, B = c.assemble(k, 1.0 / k, np.eye(n, dtype=np.complex128), _lib.FP64, want_matrix=False)
        _, b = c.assemble(k, 1.0 / k, q, _lib.FP64, want_matrix=False)
    ref = B.astype(np.clongdouble) @ q.astype(np.clongdouble)
    assert _distance(b, ref) <= U / np.sqrt(3.0) * np.sqrt(16.0 + n / 32.0)


def test_field_sums():
    """A field whose terms all have one sign and about one size (no pressure,
    positive Neumann data, a wavenumber near zero), at so many points that a warp
    sums a quarter of the sources by itself: m additions to a sum that grows
    with them have an error of sqrt(m / 3) roundings in rms relative to it, of u /
    sqrt(3) at most each, and the four warps' errors are independent.  Four
    sources make one addition."""
    mesh = M.rounded_box_enclosure(5228, seed=5228)
    S, R, k = 6 * mesh.num_faces, 16, 1e-3
    rng = np.random.default_rng(1)
    q = rng.uniform(0.5, 1.5, (mesh.num_faces, R)) + 0j
    x = M.fibonacci_sphere(32 * 148 * 3, 2.0)
    with _lib.Context(0) as c:
        c.set_mesh(mesh.vertices, mesh.faces, 4, 4)
        got = c.field(k, x, np.zeros((mesh.num_vertices, R), complex), q)
    rule, w = oracle.triangle_rule(4)
    tri = np.asarray(mesh.vertices).astype(np.longdouble)[np.asarray(mesh.faces)]
    y = np.einsum("qa,fad->fqd", np.column_stack([1 - rule.sum(axis=1), rule]).astype(np.longdouble), tri)
    normal = np.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
    weight = np.sqrt((normal * normal).sum(axis=1))[:, None] * w.astype(np.longdouble)
    at = np.arange(0, len(x), len(x) // 25)
    ref = []
    for m in at:
        r = np.sqrt(((y - x[m].astype(np.longdouble)) ** 2).sum(axis=2))
        g = weight / (4 * np.arctan2(np.longdouble(0), np.longdouble(-1)) * r)
        ref.append([-((g * np.cos(k * r)).sum(axis=1) @ q.real.astype(np.longdouble)),
                    -((g * np.sin(k * r)).sum(axis=1) @ q.real.astype(np.longdouble))])
    ref = np.array(ref)
    error = got[at].real - ref[:, 0]
    assert np.linalg.norm(error.astype(float)) <= \
        U / np.sqrt(3.0) * np.sqrt(S / 16 / 3) / 2 * np.linalg.norm(ref[:, 0].astype(float))
