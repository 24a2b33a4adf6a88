"""A linear solver that outlives its assembler: another assembler, which may get the old one's address, is another system."""
import numpy as np
import pytest

import ikarus_gb300 as ikr
from ikarus_gb300 import problems

pytestmark = pytest.mark.gpu


def _system(shape, E):
    p = problems.cantilever(*shape, L=float(shape[0]), E=E)
    fes, asm = problems.build_gpu(p)
    asm.matrix(ikr.FERequirements(fes), dbc=ikr.DBCOption.Full, export=False)
    return p, fes, asm


def test_a_new_assembler_has_to_be_factorized():
    ls = ikr.LinearSolver(rtol=1e-12)
    for k in range(8):
        p, fes, asm = _system((6, 2, 2), 1000.0 + k)
        b = np.random.default_rng(k).standard_normal(p.n_dofs) * (p.fixed == 0)
        with pytest.raises(ikr.IkarusError, match="INVALID_STATE"):
            ls.solve(asm, b)
        ls.compute(asm)
        ls.solve(asm, b)
        del asm, fes


@pytest.mark.parametrize("slabs", [0, 3])
def test_systems_of_changing_size(slabs):
    """The same solver over beams of other sizes and of the same number of nodes, with a plan or a coarse space for each."""
    ls = ikr.LinearSolver(rtol=1e-12)
    if slabs:
        ls.set_coarse_space(slabs)
    for k, shape in enumerate([(24, 2, 2), (12, 2, 2), (12, 2, 2), (9, 4, 2), (18, 7, 3), (24, 2, 2)]):
        p, fes, asm = _system(shape, 1000.0 * (k + 1))
        b = np.random.default_rng(k).standard_normal(p.n_dofs) * (p.fixed == 0)
        ls.compute(asm)
        x = np.asarray(ls.solve(asm, b))
        K = asm.matrix(ikr.FERequirements(fes), dbc=ikr.DBCOption.Full)
        # the recursive residual is at 1e-12 of b; rounding of K x adds eps |K| |x|
        bound = 1e-12 * np.linalg.norm(b) + 8 * np.sqrt(ls.last_info()[0]) * 2.0**-53 * np.linalg.norm(abs(K) @ abs(x))
        assert np.linalg.norm(K @ x - b) <= bound
        del asm, fes
