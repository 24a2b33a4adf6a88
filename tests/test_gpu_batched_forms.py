"""Which form of the batched CG the planner's choice runs: groups of the one-reduction CG from the start (in one launch or in
two), groups that take over once few enough instances are left, or the kernels of batched.cu."""
import numpy as np
import pytest

import ikarus_gb300 as ikr
from ikarus_gb300 import problems

pytestmark = pytest.mark.gpu

# instances, elements along the beam, elements across, form (152 SMs)
CASES = [
    (3, (3, 6), (1, 2), "groups"),
    (140, (12, 12), (8, 8), "groups"),    # 1 053 rows: in FP64 two launches of half the instances, two CTAs each
    (160, (1, 2), (1, 1), "two launches"),
    (300, (1, 9), (1, 2), "two launches"),
    (400, (1, 9), (1, 2), "taken over"),  # more than two launches hold
    (1, (60, 60), (16, 16), "none"),      # 17 629 rows: the vectors do not fit shared memory
]


def _run(bp, precision, variant):
    fes, asm = problems.build_gpu_batched(bp, precision=precision)
    st = ikr.NRSettings(tol=1e-9, maxIter=40, relative=True, linear_rtol=1e-3 if precision else 1e-11)
    nr = ikr.NewtonRaphson(asm, ikr.NewtonRaphsonConfig(st, ikr.LinearSolver(ikr.SolverTypeTag.gpu_PCG_Batched)))
    nr.set_batched_cg(variant=variant, first_chunk=8)
    req = ikr.FERequirements(fes)
    req.insertParameter(1.0 / 3.0)
    info = nr.solve(req)
    assert info.success and (nr.instance_info()[2] == 1).all()
    return nr, info, req.globalSolution()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,nx,nyz,form", CASES)
def test_the_form_that_runs(precision, n, nx, nyz, form):
    """Displacements against the row loop: each run ends at ||R|| <= 1e-9 ||R0||, within 1e-8 of the solution."""
    bp = problems.batched_cantilevers(n=n, seed=5, nx=nx, nyz=nyz, E=(1e3, 1e4), t=(0.1, 0.5), load_steps=3)
    nr, info, u = _run(bp, precision, -1)
    started, taken, continued = nr.batched_cg_group_launches().tolist()
    total = nr.batched_cg_launches()
    if form == "none":
        assert started == taken == continued == 0
    elif form == "taken over":
        # no group starts a solve while all instances are in it; instances are left out of later solves as they converge
        assert taken > 0 and started + taken + continued < total
    else:
        assert taken == 0 and started + continued == total and started >= info.iterations
        if form == "two launches":
            assert started > info.iterations
    row_loop, _, v = _run(bp, precision, 0)
    assert (row_loop.batched_cg_group_launches() == 0).all()
    for a, b in zip(bp.node_offsets[:-1], bp.node_offsets[1:]):
        assert np.abs(u[3 * a:3 * b] - v[3 * a:3 * b]).max() <= 2e-8 * np.abs(u[3 * a:3 * b]).max()
