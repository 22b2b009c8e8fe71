"""The zero-lag gradient against the FP64 oracle over shot counts (one to several elements
a block), box and distorted elements, and both stress forms.  Bar: relative L2 1e-10."""
import numpy as np
import pytest

import oracle as O
from problems import RHO, rel_l2, tiny, traces_from_history
from test_gpu_line import _distorted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nshot,distorted,lambda_2mu", [(1, True, False), (2, False, True), (3, False, False), (4, True, True),
                                                        (5, False, True), (6, True, False), (7, False, False), (8, False, True)])
def test_gradient_matches_oracle(gpu_lib, nshot, distorted, lambda_2mu):
    from hirensi_b200.solver import Solver
    p = tiny(nshot=nshot, nstep=25)
    mesh = _distorted(p["mesh"]) if distorted else p["mesh"]
    om = O.OracleMesh(mesh, RHO)
    S = O.OracleSystem.assemble(om, p["lam"], p["mu"])
    dis = 1e-6 * np.random.default_rng(5).standard_normal((nshot, len(p["eqdis"]), p["nstep"] + 1))
    with Solver("fp64") as s:
        s.set_mesh(mesh, RHO)
        s.assemble(p["lam"], p["mu"])
        s.set_history(mesh.store_eq)
        s.set_shots(p["nstep"], p["dt"], p["src_eq"], p["src_b"], p["ftab"])
        s.set_receivers(p["eqdis"], p["eqdis_map"])
        s.forward()
        gl, gm = s.adjoint_gradient(dis, lambda_2mu=lambda_2mu)
    rl, rm = np.zeros(mesh.nj), np.zeros(mesh.nj)
    for k in range(nshot):
        b = np.zeros(mesh.neq)
        b[p["src_eq"][k]] = 1.0
        h = S.forward(b, p["ftab"][k], p["nstep"], p["dt"], mesh.store_eq, 1)
        pk = S.adjoint(p["nstep"], p["dt"], mesh.store_eq, h, p["eqdis"], p["eqdis_map"], dis[k])
        a, c = O.control(om, p["nstep"], p["dt"], mesh.store_eq, h, pk, lambda_2mu=lambda_2mu)
        rl += a
        rm += c
    assert rel_l2(gl, rl) < 1e-10 and rel_l2(gm, rm) < 1e-10
