"""Gathered tangents of more elements than are held at a time: the sums over the parts are those of one part, bit for bit."""
import numpy as np
import pytest

import ikarus_gb300 as ikr
from ikarus_gb300 import problems

pytestmark = pytest.mark.gpu

FORMS = [  # precision, material, eas, n_eas, FP32 tangent kernel
    (0, 0, 0, 0, 0),   # FP64 element blocks
    (0, 1, 0, 0, 0),   # FP64 element matrices
    (1, 0, 0, 0, 3),   # FP32 element blocks
    (0, 0, 1, 9, 0),
    (1, 0, 2, 9, 0),   # FP64 element matrices, FP32 values: rounded once
]


@pytest.mark.parametrize("part", [1, 7, 44, 45])
@pytest.mark.parametrize("precision,material,eas,n_eas,kernel", FORMS)
def test_parts_do_not_change_the_tangent(precision, material, eas, n_eas, kernel, part):
    """45 elements, nodes and elements in random order: single elements, ragged parts, all but one, all."""
    p = problems.cantilever(5, 3, 3, L=5.0, jitter=0.1, seed=3, eas=eas, n_eas=n_eas)
    p.material = material
    rng = np.random.default_rng(4)
    new, order = rng.permutation(p.mesh.n_nodes), rng.permutation(p.mesh.n_elems)
    coords, fixed = np.empty_like(p.mesh.coords), np.empty_like(p.fixed.reshape(-1, 3))
    coords[new], fixed[new] = p.mesh.coords, p.fixed.reshape(-1, 3)
    p.mesh.coords, p.fixed = coords, fixed.reshape(-1)
    p.mesh.conn = new[p.mesh.conn[order]].astype(np.int32)
    p.face_elem = np.argsort(order)[p.face_elem].astype(np.int32)
    fes, asm = problems.build_gpu(p, precision=precision)
    if n_eas:
        fes.alpha = 1e-4 * rng.standard_normal((p.mesh.n_elems, n_eas))
    if kernel:
        asm.set_tangent_kernel(kernel)
    req = ikr.FERequirements(fes, 0.005 * rng.standard_normal(p.n_dofs), 0.6)
    for dbc in (ikr.DBCOption.Full, ikr.DBCOption.Raw, ikr.DBCOption.Reduced):
        asm.set_gather_part(0)
        whole = asm.matrix(req, dbc=dbc).data.copy()
        asm.set_gather_part(part)
        assert np.array_equal(asm.matrix(req, dbc=dbc).data, whole)
