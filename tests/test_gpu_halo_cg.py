"""The one-reduction persistent CG (CG kinds 12 and 13): every split of the rows over the CTAs (chunks of 4, 8 and 16
rows, whole slices, matrix resident in shared memory or streamed), at the sizes where the split changes, on structured
and shuffled node numberings, against the other persistent form and the true residual."""
import numpy as np
import pytest

from ikarus_gb300 import problems

pytestmark = pytest.mark.gpu

# elements per direction of a clamped block; the nodes are 8, 608, 609, 1 216, 1 224, 2 432, 2 511 (the chunks change
# above 4, 8 and 16 rows per SM of 152), then 14 161 and 25 947 (resident in FP32, streamed in FP64), 48 000 (streamed)
SIZES = [(1, 1, 1), (18, 7, 3), (28, 6, 2), (18, 7, 7), (16, 7, 8), (18, 15, 7), (30, 8, 8), (48, 16, 16),
         (60, 20, 20)]


def block(shape, fp32, shuffle=False, seed=0):
    p = problems.eas_block(*shape, nu=0.3, eas=0, n_eas=0)
    if shuffle:
        perm = np.random.default_rng(seed).permutation(p.mesh.n_nodes)
        coords = np.empty_like(p.mesh.coords)
        coords[perm] = p.mesh.coords
        p.mesh.coords = coords
        p.mesh.conn = perm[p.mesh.conn].astype(np.int32)
        fixed = np.empty_like(p.fixed).reshape(-1, 3)
        fixed[perm] = p.fixed.reshape(-1, 3)
        p.fixed = fixed.reshape(-1)
    fes, asm = problems.build_gpu(p, precision=fp32)
    return p, fes, asm


def solve(ikr, asm, kind, b, rtol, keep=0.3):
    ls = ikr.LinearSolver(ikr.SolverTypeTag.gpu_PCG_BlockJacobi, rtol=rtol, max_iter=20000)
    ls.set_kernel(kind, keep)
    ls.compute(asm)
    x = ls.solve(asm, b)
    it, rel = ls.last_info()
    assert np.array_equal(x, ls.solve(asm, b)), "repeated solve is not bit-identical"
    assert rel <= rtol
    return x, it


@pytest.mark.parametrize("shape", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("fp32", [0, 1], ids=["fp64", "fp32"])
def test_halo_cg_solves_at_every_split(ikr, shape, fp32):
    p, fes, asm = block(shape, fp32)
    req = ikr.FERequirements(fes, 0.002 / max(shape) * np.random.default_rng(1).standard_normal(p.n_dofs)
                             * (p.fixed == 0), 1.0)
    K = asm.matrix(req, dbc=ikr.DBCOption.Full)
    b = np.random.default_rng(0).standard_normal(p.n_dofs) * (p.fixed == 0)
    rtol, eps = (1e-5, 2.0**-24) if fp32 else (1e-11, 2.0**-53)
    for kind in (12, 13):
        x, it = solve(ikr, asm, kind, b, rtol)
        # the recursive residual is at the tolerance; each of its updates rounds by eps |K| |x|, a random walk over
        # the iterations
        bound = rtol * np.linalg.norm(b) + 8 * np.sqrt(it) * eps * np.linalg.norm(abs(K) @ abs(x))
        assert np.linalg.norm(K @ x - b) <= bound
    ref, it_ref = solve(ikr, asm, 7, b, rtol)
    # the same recurrences: the iteration counts differ by what rounding moves the last ones
    assert abs(it - it_ref) <= 2 + 0.1 * it_ref


@pytest.mark.parametrize("fp32", [0, 1], ids=["fp64", "fp32"])
def test_shuffled_numbering(ikr, fp32):
    """A shuffled numbering makes every CTA's halo almost the whole system."""
    p, fes, asm = block((20, 9, 9), fp32, shuffle=True)
    req = ikr.FERequirements(fes)
    K = asm.matrix(req, dbc=ikr.DBCOption.Full)
    b = np.random.default_rng(0).standard_normal(p.n_dofs) * (p.fixed == 0)
    rtol, eps = (1e-5, 2.0**-24) if fp32 else (1e-11, 2.0**-53)
    x, it = solve(ikr, asm, 12, b, rtol)
    bound = rtol * np.linalg.norm(b) + 8 * np.sqrt(it) * eps * np.linalg.norm(abs(K) @ abs(x))
    assert np.linalg.norm(K @ x - b) <= bound


def test_without_a_split_that_fits_the_classic_kernel_runs(ikr):
    """A shuffled numbering of 92 k rows: halos of more than 12 k rows, so kind 12 runs the kernel of kind 7."""
    p, fes, asm = block((96, 30, 30), 1, shuffle=True)
    req = ikr.FERequirements(fes)
    asm.matrix(req, dbc=ikr.DBCOption.Full, export=False)
    b = np.random.default_rng(0).standard_normal(p.n_dofs) * (p.fixed == 0)
    x, it = solve(ikr, asm, 12, b, 1e-4)
    ref, it_ref = solve(ikr, asm, 7, b, 1e-4)
    assert it == it_ref and np.array_equal(x, ref)


def test_wait_that_runs_out(ikr):
    """CTA 0 withholds its first sums: every CTA's wait runs out, the solve reports it and the handle recovers."""
    p, fes, asm = block((18, 7, 3), 0)
    req = ikr.FERequirements(fes)
    asm.matrix(req, dbc=ikr.DBCOption.Full, export=False)
    b = np.random.default_rng(0).standard_normal(p.n_dofs) * (p.fixed == 0)
    ls = ikr.LinearSolver(ikr.SolverTypeTag.gpu_PCG_BlockJacobi, rtol=1e-10)
    ls.set_kernel(12, 0.0)
    ls.compute(asm)
    ref = ls.solve(asm, b)
    ls.set_wait_test(barrier_polls=4096, withhold_first_arrival=True)
    with pytest.raises(ikr.IkarusError, match="TIMEOUT"):
        ls.solve(asm, b)
    assert np.array_equal(ls.solve(asm, b), ref)


def test_non_finite_right_hand_side_breaks_down(ikr):
    p, fes, asm = block((4, 2, 2), 0)
    req = ikr.FERequirements(fes)
    asm.matrix(req, dbc=ikr.DBCOption.Full, export=False)
    ls = ikr.LinearSolver(ikr.SolverTypeTag.gpu_PCG_BlockJacobi, rtol=1e-10)
    ls.set_kernel(12, 0.0)
    ls.compute(asm)
    b = np.zeros(p.n_dofs)
    assert np.array_equal(ls.solve(asm, b), b)
    b[-1] = np.nan
    with pytest.raises(ikr.IkarusError, match="CG_BREAKDOWN"):
        ls.solve(asm, b)
