"""Batched instances in other units: stiffness and loads times a power of two give the same displacements."""
import numpy as np
import pytest

import ikarus_gb300 as ikr
from ikarus_gb300 import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [-42, 80])
@pytest.mark.parametrize("n", [3, 140])
def test_units_of_force_do_not_matter(n, exponent):
    """FP32 tangents and CG: nodal residuals around 1e-24 (at the end of the Newton iteration) or 1e22 have squares outside the
    range of FP32, so r.r has to be summed in a wider one; r.z and p.q, smaller or larger by the stiffness, stay inside.
    Forces, tangents and scalars scale exactly as far as nothing under- or overflows: the displacements agree to 2e-8
    (both runs end at ||R|| <= 1e-9 ||R0||)."""
    us, its = [], []
    for f in (1.0, 2.0**exponent):
        bp = problems.batched_cantilevers(n=n, seed=5, nx=(4, 6), nyz=(2, 2), E=(1e3, 1e4), t=(0.1, 0.5), load_steps=3)
        bp.lam_e, bp.mu_e, bp.face_traction = bp.lam_e * f, bp.mu_e * f, bp.face_traction * f
        fes, asm = problems.build_gpu_batched(bp, precision=1)
        st = ikr.NRSettings(tol=1e-9, maxIter=40, relative=True, linear_rtol=1e-3)
        nr = ikr.NewtonRaphson(asm, ikr.NewtonRaphsonConfig(st, ikr.LinearSolver(ikr.SolverTypeTag.gpu_PCG_Batched)))
        req = ikr.FERequirements(fes)
        req.insertParameter(1.0 / 3.0)
        assert nr.solve(req).success
        us.append(req.globalSolution())
        its.append(nr.instance_linear_iterations())
    # a sum that under- or overflows ends solves early or not at all (one instance may take a Newton iteration more)
    assert abs(its[1].sum() - its[0].sum()) <= 0.1 * its[0].sum()
    for a, b in zip(bp.node_offsets[:-1], bp.node_offsets[1:]):
        u, v = us[0][3 * a:3 * b], us[1][3 * a:3 * b]
        assert np.abs(u - v).max() <= 2e-8 * np.abs(u).max()
