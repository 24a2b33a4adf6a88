"""The planner's choice of the batched CG (the one-reduction kernel with a group of CTAs per instance where the split fits)
against the row loop (variant 0), at the sizes where the split, the layout or the fallback changes."""
import numpy as np
import pytest

import ikarus_gb300 as ikr
from ikarus_gb300 import problems

pytestmark = pytest.mark.gpu

# instances, elements along the beam, elements across (lowest, highest), nodes of each instance renumbered at random
CASES = [
    (1, (30, 30), (5, 5), False),   # 1 116 rows over 35 CTAs, everything resident
    (1, (30, 30), (5, 5), True),    # columns of a row all over the instance: halos of several hundred rows
    (9, (1, 2), (1, 1), False),     # 8 or 12 rows: several instances in a slice of 32 rows
    (2, (8, 9), (3, 4), False),     # slices split unevenly, the first and the last shared
    (140, (4, 4), (6, 6), False),   # one CTA each, blocks streamed, one pass over 245 rows
    (140, (6, 6), (8, 8), False),   # 567 rows: two passes in FP32, three in FP64
    (140, (12, 12), (8, 8), False), # 1 053 rows: three passes in FP32; FP64 does not fit and keeps the row loop
    (160, (1, 2), (1, 1), False),   # more instances than SMs: no split
    (300, (1, 9), (1, 2), False),   # no split at first, then the instances left over are taken over
]


def _problem(n, nx, nyz, shuffled):
    bp = problems.batched_cantilevers(n=n, seed=5, nx=nx, nyz=nyz, E=(1e3, 1e4), t=(0.1, 0.5), load_steps=3)
    if shuffled:
        rng = np.random.default_rng(2)
        new = np.concatenate([a + rng.permutation(b - a) for a, b in zip(bp.node_offsets[:-1], bp.node_offsets[1:])])
        coords, fixed = np.empty_like(bp.mesh.coords), np.empty_like(bp.fixed.reshape(-1, 3))
        coords[new], fixed[new] = bp.mesh.coords, bp.fixed.reshape(-1, 3)
        bp.mesh.coords, bp.mesh.conn, bp.fixed = coords, new[bp.mesh.conn].astype(np.int32), fixed.reshape(-1)
    return bp


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,nx,nyz,shuffled", CASES)
def test_split_instances_match_the_row_loop(precision, n, nx, nyz, shuffled):
    """One load increment, in launches of 40 iterations and more so that every solve is split several times.  Each run
    ends at ||R|| <= 1e-9 ||R0||, where the displacements are within 1e-8 of the solution: 2e-8 between the two."""
    bp = _problem(n, nx, nyz, shuffled)
    us = []
    for variant in (0, -1):
        fes, asm = problems.build_gpu_batched(bp, precision=precision)
        st = ikr.NRSettings(tol=1e-9, maxIter=40, relative=True, linear_rtol=1e-3 if precision else 1e-11)
        nr = ikr.NewtonRaphson(asm, ikr.NewtonRaphsonConfig(st, ikr.LinearSolver(ikr.SolverTypeTag.gpu_PCG_Batched)))
        nr.set_batched_cg(variant=variant, first_chunk=40)
        req = ikr.FERequirements(fes)
        req.insertParameter(1.0 / 3.0)
        assert nr.solve(req).success
        assert (nr.instance_info()[2] == 1).all()
        us.append(req.globalSolution())
    for a, b in zip(bp.node_offsets[:-1], bp.node_offsets[1:]):
        u, v = us[0][3 * a:3 * b], us[1][3 * a:3 * b]
        assert np.abs(u - v).max() <= 2e-8 * np.abs(u).max()


@pytest.mark.parametrize("precision", [0, 1])
def test_iteration_limit_and_zero_right_hand_side(precision):
    """A solve that reaches its limit leaves the iterate of exactly that many iterations, and an unloaded instance is
    left alone."""
    bp = problems.batched_cantilevers(n=3, seed=3, nx=(4, 6), nyz=(2, 2), E=(1e3, 1e3), t=(0.2, 0.3), load_steps=1)
    bp.face_traction[bp.face_elem < bp.elem_offsets[1]] = 0.0
    its = []
    for variant in (0, -1):
        fes, asm = problems.build_gpu_batched(bp, precision=precision)
        st = ikr.NRSettings(tol=1e-9, maxIter=2, relative=True, linear_rtol=1e-12, linear_max_iter=7)
        nr = ikr.NewtonRaphson(asm, ikr.NewtonRaphsonConfig(st, ikr.LinearSolver(ikr.SolverTypeTag.gpu_PCG_Batched)))
        nr.set_batched_cg(variant=variant, first_chunk=7)
        req = ikr.FERequirements(fes)
        req.insertParameter(1.0)
        nr.solve(req)
        its.append(nr.instance_linear_iterations().tolist())
        u = req.globalSolution()
        assert (u[:3 * bp.node_offsets[1]] == 0).all() and (u[3 * bp.node_offsets[1]:] != 0).any()
    assert its[0] == its[1] == [0, 14, 14]
