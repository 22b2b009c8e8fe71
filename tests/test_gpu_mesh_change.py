"""A context whose mesh is set again: everything that was derived from the old mesh goes."""
import dataclasses

import numpy as np
import pytest

from problems import RHO, tiny

pytestmark = pytest.mark.gpu


def _shots(s, p, mesh):
    s.set_history(mesh.store_eq)
    s.set_shots(p["nstep"], p["dt"], p["src_eq"], p["src_b"], p["ftab"])
    s.set_receivers(p["eqdis"], p["eqdis_map"])


@pytest.mark.parametrize("matrix_free", [False, True])
def test_elements_in_another_order(gpu_lib, matrix_free):
    """The same equations with the elements listed in another order: DIAG_M, C, K, G and
    the seismograms are those of a context that only ever saw the second mesh."""
    from hirensi_b200.solver import Solver
    p = tiny(nshot=2, nstep=30)
    mesh = p["mesh"]
    perm = np.random.default_rng(5).permutation(mesh.nel)
    other = dataclasses.replace(mesh, inod=mesh.inod[perm], mtel=mesh.mtel[perm], eid=mesh.eid[perm])
    out = []
    for meshes in ((mesh, other), (other,)):
        with Solver("fp64") as s:
            for m in meshes:
                s.set_mesh(m, RHO)
                s.set_operator_mode(matrix_free)
                s.assemble(p["lam"], p["mu"])
            _shots(s, p, other)
            s.set_variant(96, 96)
            s.forward()
            ops = [] if matrix_free else [s.operator_csr(w)[2] for w in range(3)]
            out.append([s.diag_m(), s.traces()] + ops)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
