"""Assembly from element vectors and matrices by ordered gathers, at the element counts and numberings where the work per
block, the Gauss-point butterflies or the gather lists change."""
import numpy as np
import pytest

import oracle
import ikarus_gb300 as ikr
from ikarus_gb300 import problems

pytestmark = pytest.mark.gpu

# elements: fewer than a warp holds (4), one more, a remainder in every block size, and more than 4 096 (larger blocks)
MESHES = [(1, 1, 1), (3, 1, 1), (5, 1, 1), (3, 3, 3), (11, 3, 1), (17, 17, 15)]


def _problem(n, shuffled, material=0, eas=0, n_eas=0):
    p = problems.cantilever(*n, L=float(n[0]), jitter=0.1, seed=3, eas=eas, n_eas=n_eas)
    p.material = material
    if shuffled:  # nodes renumbered, elements in another order
        rng = np.random.default_rng(4)
        new, order = rng.permutation(p.mesh.n_nodes), rng.permutation(p.mesh.n_elems)
        coords, fixed = np.empty_like(p.mesh.coords), np.empty_like(p.fixed.reshape(-1, 3))
        coords[new], fixed[new] = p.mesh.coords, p.fixed.reshape(-1, 3)
        p.mesh.coords, p.fixed = coords, fixed.reshape(-1)
        p.mesh.conn = new[p.mesh.conn[order]].astype(np.int32)
        p.face_elem = np.argsort(order)[p.face_elem].astype(np.int32)
    return p


def _compare(p, alpha=None, precision=0, rtol=1e-12):
    """FP64: within 1e-12 of the oracle, relative to the largest entry; the pattern is exact.  rtol: the matrix."""
    fes, asm = problems.build_gpu(p, precision=precision)
    o = oracle.from_problem(p)
    u = 0.02 / max(p.mesh.shape[1:]) * np.random.default_rng(6).standard_normal(p.n_dofs)
    if alpha is not None:
        fes.alpha = alpha
        o.alpha = alpha
    req = ikr.FERequirements(fes, u, 0.6)
    for dbc, odbc in ((ikr.DBCOption.Full, oracle.DBC_FULL), (ikr.DBCOption.Raw, oracle.DBC_RAW),
                      (ikr.DBCOption.Reduced, oracle.DBC_REDUCED)):
        r = o.assemble_vector(u, 0.6, odbc)
        assert np.abs(asm.vector(req, dbc=dbc) - r).max() <= 1e-12 * np.abs(r).max()
        cp, ri, v, n = o.assemble_matrix_csc(u, 0.6, odbc)
        K = asm.matrix(req, dbc=dbc)
        assert np.array_equal(K.indptr, cp) and np.array_equal(K.indices, ri)
        assert np.abs(K.data - v).max() <= rtol * np.abs(v).max()


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("n", MESHES)
def test_displacement_elements(n, shuffled):
    _compare(_problem(n, shuffled))


@pytest.mark.parametrize("material", [1, 2])
def test_other_materials(material):
    _compare(_problem((5, 3, 2), True, material))


@pytest.mark.parametrize("precision,rtol", [(0, 1e-12), (1, 1e-6)])
@pytest.mark.parametrize("kind,n_eas", [(1, 9), (1, 21), (2, 9), (3, 9)])
@pytest.mark.parametrize("n", [(1, 1, 1), (5, 1, 1), (3, 3, 3)])
def test_enhanced_strain_elements(n, kind, n_eas, precision, rtol):
    """FP32 assemblers hold the matrix, formed in FP64, to 1e-6."""
    p = _problem(n, True, 0, kind, n_eas)
    scale = 1e-4 if kind == 1 else 5e-3  # of the modes: strains over an element's size, or displacement gradients
    _compare(p, scale * np.random.default_rng(8).standard_normal((p.mesh.n_elems, n_eas)), precision, rtol)


@pytest.mark.parametrize("slabs", [3, 16])
@pytest.mark.parametrize("n", [(40, 3, 3), (64, 7, 5)])
def test_coarse_operator_of_ragged_slabs(n, slabs):
    """A_c = P^T K P over runs of 256 nodes that end inside a slab, nodes numbered at random: with the correction, a solve
    to 1e-11 gives the plain solver's solution to 1e-8 in fewer iterations."""
    p = _problem(n, True)
    fes, asm = problems.build_gpu(p)
    req = ikr.FERequirements(fes, None, 1.0)
    asm.matrix(req, dbc=ikr.DBCOption.Full, export=False)
    b = np.random.default_rng(9).standard_normal(p.n_dofs) * (1 - p.fixed)
    xs, its = [], []
    for k in (0, slabs):
        ls = ikr.LinearSolver(rtol=1e-11, max_iter=20000)
        if k:
            ls.set_coarse_space(k)
        ls.compute(asm)
        xs.append(np.asarray(ls.solve(asm, b)))
        its.append(ls.last_info()[0])
    assert np.abs(xs[1] - xs[0]).max() <= 1e-8 * np.abs(xs[0]).max()
    assert its[1] < its[0]
