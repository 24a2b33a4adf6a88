"""Two right-hand sides with one FP32 tangent: the two-barrier kinds solve both in one launch, the one-reduction kind one after
the other."""
import numpy as np
import pytest

import oracle
from ikarus_gb300 import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,multi,one_launch", [(5, True, True), (7, True, True), (7, False, False),
                                                   (12, True, False), (-1, True, False)])
def test_arc_length_by_kind(ikr, kind, multi, one_launch):
    """The path of the FP64 oracle: load factors to 1e-6 and the displacement to 1e-5 of the largest entry, as for every mixed
    form (tests/test_gpu_path_following.py)."""
    p = problems.cantilever(8, 2, 2, traction=(0.0, 0.0, -0.5), load_steps=4)
    o = oracle.from_problem(p)
    u0 = np.zeros(p.n_dofs)
    s = 0.25 * np.sqrt(2.0) * np.linalg.norm(np.linalg.solve(o.assemble_matrix_dense(u0, 1.0), o.assemble_vector(u0, 1.0)))
    ref = oracle.from_problem(p).path_following(4, s, tol=1e-10, max_iter=30)
    fes, asm = problems.build_gpu(p, precision=1)
    req = ikr.FERequirements(fes)
    ls = ikr.LinearSolver(rtol=1e-13)
    ls.set_kernel(kind, -1.0 if kind < 0 else 0.0)
    ls.set_multi_rhs(multi)
    st = ikr.NRSettings(tol=1e-10, maxIter=60, eisenstat_walker=True, linear_rtol=1e-2, linear_rtol_min=1e-7)
    nr = ikr.NewtonRaphson(asm, ikr.NewtonRaphsonConfig(st, ls))
    pf = ikr.PathFollowing(nr, 4, s, ikr.ArcLength())
    assert pf.run(req).success
    together, separate = ls.multi_rhs_info()
    assert (together > 0 and separate == 0) if one_launch else (together == 0 and separate > 0)
    assert abs(req.parameter() - ref["lam"]) <= 1e-6 * abs(ref["lam"])
    assert np.abs(req.globalSolution() - ref["u"]).max() <= 1e-5 * np.abs(ref["u"]).max()
