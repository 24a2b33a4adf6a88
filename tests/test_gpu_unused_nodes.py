"""Clamped nodes that no element uses: their rows of the tangent are the identity (Full Dirichlet treatment) wherever they
sit in the slices of 32 rows, so the systems around them are solved as without them."""
import numpy as np
import pytest
import scipy.sparse.linalg as spla

from ikarus_gb300 import problems

pytestmark = pytest.mark.gpu

# 36 nodes of the mesh take a slice and four rows: unused nodes in the second slice, two slices of them behind, one slice
# and one row in front
PLACES = {"same_slice": (0, 3), "slices_behind": (0, 70), "slices_in_front": (33, 0)}


def _padded(p, front, behind):
    """The problem with unused clamped nodes in front of and behind its own."""
    c, n = p.mesh.coords, front + behind
    far = 20.0 + np.arange(3.0 * n).reshape(n, 3)
    p.mesh.coords = np.concatenate([far[:front], c, far[front:]])
    p.mesh.conn = (p.mesh.conn + front).astype(np.int32)
    one = np.ones(3 * n, dtype=p.fixed.dtype)
    p.fixed = np.concatenate([one[:3 * front], p.fixed, one[3 * front:]])
    return p


@pytest.mark.parametrize("place", PLACES)
@pytest.mark.parametrize("precision,eas,n_eas,path", [(0, 0, 0, 0), (0, 1, 9, 0), (1, 1, 9, 0), (1, 0, 0, 1),
                                                      (1, 0, 0, 2), (1, 0, 0, 3)])
def test_rows_without_elements_are_solved(ikr, place, precision, eas, n_eas, path):
    """path: the FP32 tangent's kernels.  The solutions agree to the tolerance of the solves times the condition number
    (under 1e4), the unused rows to the tolerance."""
    front, behind = PLACES[place]
    rng = np.random.default_rng(3)
    plain = problems.cantilever(3, 2, 2, L=3.0, eas=eas, n_eas=n_eas)
    n = plain.n_dofs
    fes, asm = problems.build_gpu(plain, precision=0)
    K = asm.matrix(ikr.FERequirements(fes), dbc=ikr.DBCOption.Full)
    b = rng.standard_normal(n + 3 * (front + behind))
    own = slice(3 * front, 3 * front + n)
    b[own][plain.fixed != 0] = 0.0
    x_own = spla.spsolve(K.tocsc(), b[own])
    p = _padded(problems.cantilever(3, 2, 2, L=3.0, eas=eas, n_eas=n_eas), front, behind)
    fes, asm = problems.build_gpu(p, precision=precision)
    if path:
        asm.set_tangent_kernel(path)
    req = ikr.FERequirements(fes)
    asm.matrix(req, dbc=ikr.DBCOption.Full, export=False)
    rtol = 1e-6 if precision else 1e-12
    for kind in (7, 12):
        ls = ikr.LinearSolver(ikr.SolverTypeTag.gpu_PCG_BlockJacobi, rtol=rtol, max_iter=2000)
        ls.set_kernel(kind, 0.0)
        ls.compute(asm)
        x = np.asarray(ls.solve(asm, b))
        rest = np.delete(x - b, np.r_[own])
        assert np.abs(x[own] - x_own).max() <= 1e4 * rtol * np.abs(x_own).max()
        assert np.abs(rest).max() <= 100 * rtol * np.abs(b).max()
