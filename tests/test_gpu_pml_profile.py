"""Stretching profiles of either sign assemble as the oracle does; only a node past the top
face is refused.  Bar: 1e-14 of the largest entry (the elements add in another order)."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from hirensi_b200.mesh import box_mesh
from problems import RHO, layered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("matrix_free", [False, True])
def test_negative_stretching_factors(gpu_lib, matrix_free):
    from hirensi_b200.solver import Solver
    mesh = box_mesh(3, 2, 2, 2.5, 1, alpha0=-3.0)   # factors 1, 0.25 and -2 across the layer
    lam, mu = layered(mesh)
    S = O.OracleSystem.assemble(O.OracleMesh(mesh, RHO), lam, mu)
    with Solver("fp64") as s:
        s.set_mesh(mesh, RHO)
        s.set_operator_mode(matrix_free)
        s.assemble(lam, mu)
        d = s.diag_m()
        ops = [] if matrix_free else [s.operator_csr(w) for w in range(3)]
    ref = S.vectors()[0]
    assert ref.min() < 0 and np.max(np.abs(d - ref)) <= 1e-14 * np.abs(ref).max()
    for w, (ia, ja, a) in enumerate(ops):
        ia_r, ja_r, a_r = S.csr(w)
        assert np.array_equal(ia, ia_r) and np.array_equal(ja, ja_r)
        assert np.max(np.abs(a - a_r)) <= 1e-14 * np.abs(a_r).max()


@pytest.mark.parametrize("matrix_free", [False, True])
def test_node_past_the_top_is_refused(gpu_lib, matrix_free):
    from hirensi_b200.capi import HRN_EMESH, HrnError
    from hirensi_b200.solver import Solver
    mesh = box_mesh(2, 2, 1, 2.5, 1)
    pml = mesh.pml_param.copy()
    pml[4, 3] = -1.0   # the top zone starts below the surface
    with Solver("fp64") as s:
        s.set_mesh(dataclasses.replace(mesh, pml_param=pml), RHO)
        s.set_operator_mode(matrix_free)
        with pytest.raises(HrnError) as e:
            s.assemble(*layered(mesh))
        assert e.value.code == HRN_EMESH
