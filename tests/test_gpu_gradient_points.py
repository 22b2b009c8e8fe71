"""The gradient kernel with one thread per point (one shot; shot counts that are not a power
of two from two blocks an SM up), against the oracle's correlation of the device's own
histories.  The grids end in a block of fewer elements, and lie on either side of the rule.
Bar: relative L2 1e-10 in FP64 and in FP32 stepping (the correlation is FP64 in both)."""
import numpy as np
import pytest

import oracle as O
from problems import RHO, rel_l2, tiny
from test_gpu_line import _distorted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,nshot,precision,distorted,lambda_2mu", [
    ((1, 1, 1), 1, "fp64", False, False), ((3, 2, 1), 1, "fp32", True, True), ((15, 9, 9), 1, "fp64", True, False),
    ((15, 9, 9), 3, "fp32", True, False), ((15, 9, 9), 3, "fp64", False, True), ((15, 9, 9), 5, "fp32", False, False),
    ((15, 9, 9), 6, "fp64", True, True), ((15, 9, 9), 7, "fp32", True, False), ((13, 13, 7), 5, "fp64", False, False)])
def test_gradient_of_device_histories(gpu_lib, size, nshot, precision, distorted, lambda_2mu):
    from hirensi_b200.mesh import box_mesh
    from hirensi_b200.solver import Solver
    p = tiny(nshot=1, nstep=8, fr=900.0)
    mesh = box_mesh(*size, 2.5, 1)
    if distorted:
        mesh = _distorted(mesh)
    rng = np.random.default_rng(3)
    mu = RHO * rng.uniform(200.0, 400.0, mesh.nj) ** 2
    surf = mesh.store_nodes[np.abs(mesh.xyz[mesh.store_nodes, 2]) < 1e-9]
    rec = mesh.equations(rng.choice(surf, 5, replace=False))
    with Solver(precision) as s:
        s.set_mesh(mesh, RHO)
        s.assemble(2 * mu, mu)
        s.set_history(mesh.store_eq)
        s.set_shots(p["nstep"], p["dt"], mesh.equations(rng.choice(surf, nshot, replace=False), comps=(2,)), np.eye(nshot),
                    np.stack([p["ftab"][0]] * nshot))
        s.set_receivers(rec, mesh.store_position(rec))
        s.forward()
        gl, gm = s.adjoint_gradient(1e-6 * rng.standard_normal((nshot, rec.size, p["nstep"] + 1)), lambda_2mu=lambda_2mu, keep_p=True)
        pairs = [(s.history(k), s.adjoint_history(k)) for k in range(nshot)]
    om = O.OracleMesh(mesh, RHO)
    rl, rm = np.zeros(mesh.nj), np.zeros(mesh.nj)
    for u, q in pairs:
        a, b = O.control(om, p["nstep"], p["dt"], mesh.store_eq, u, q, lambda_2mu=lambda_2mu)
        rl, rm = rl + a, rm + b
    assert np.abs(rl).max() > 0 and np.abs(rm).max() > 0
    assert rel_l2(gl, rl) < 1e-10 and rel_l2(gm, rm) < 1e-10
