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


def test_lbfgs_memory_of_another_mesh(gpu_lib):
    """The memory is sized for the mesh it was set up on: a direction on a larger one is refused."""
    import torch
    from hirensi_b200.capi import HrnError
    from hirensi_b200.inversion import DeviceBackend
    from hirensi_b200.mesh import box_mesh
    from hirensi_b200.solver import Solver
    small, large = box_mesh(1, 1, 1, 2.5, 1), box_mesh(3, 2, 2, 2.5, 1)

    def vectors(mesh):
        v = [torch.full((mesh.nj,), float(k), dtype=torch.float64, device="cuda") for k in range(1, 12)]
        torch.cuda.synchronize()
        return v

    with Solver("fp64") as s:
        v = vectors(small)
        for again in range(2):   # set again with as many nodes: the memory stays
            s.set_mesh(small, RHO)
            back = DeviceBackend(s, small)
            if not again:
                back.lbfgs_setup(3, v[0])
            back.lbfgs_direction(2 + again, 1, *v[:10])
        w = vectors(large)
        s.set_mesh(large, RHO)
        back = DeviceBackend(s, large)
        with pytest.raises(HrnError):
            back.lbfgs_direction(4, 1, *w[:10])
        back.lbfgs_setup(3, w[0])
        back.lbfgs_direction(2, 1, *w[:10])
        torch.cuda.synchronize()


def test_lbfgs_direction_before_the_first_iteration(gpu_lib):
    """iter < iter_begin names no pair of the memory."""
    import torch
    from hirensi_b200.capi import HrnError
    from hirensi_b200.inversion import DeviceBackend
    from hirensi_b200.solver import Solver
    mesh = tiny()["mesh"]
    v = [torch.full((mesh.nj,), float(k), dtype=torch.float64, device="cuda") for k in range(1, 12)]
    torch.cuda.synchronize()
    with Solver("fp64") as s:
        s.set_mesh(mesh, RHO)
        back = DeviceBackend(s, mesh)
        back.lbfgs_setup(3, v[0])
        for it in (-1, -4, -7):
            with pytest.raises(HrnError):
                back.lbfgs_direction(it, 1, *v[:10])


@pytest.mark.parametrize("nshot,precision", [(1, "fp64"), (3, "fp64"), (4, "fp32")])
def test_mesh_set_between_forward_and_adjoint(gpu_lib, nshot, precision):
    """Checkpoints of the line operator, whose tables go with the mesh: the stored operator
    recomputes the segments.  Bars: 1e-11 between FP64 variants, 1e-4 with FP32 stepping."""
    from problems import rel_l2
    from hirensi_b200.solver import Solver
    p = tiny(nshot=nshot, nstep=30)
    dis = 1e-6 * np.random.default_rng(3).standard_normal((nshot, len(p["eqdis"]), p["nstep"] + 1))
    out = []
    for again in (False, True):
        with Solver(precision) as s:
            s.set_mesh(p["mesh"], RHO)
            s.assemble(p["lam"], p["mu"])
            _shots(s, p, p["mesh"])
            s.set_checkpointing(7)
            s.set_variant(97, 97)
            s.forward()
            states = s.state(14, 0)
            if again:
                s.set_mesh(p["mesh"], RHO)
                assert all(np.array_equal(a, b) for a, b in zip(states, s.state(14, 0)))
            g = s.adjoint_gradient(dis)
            out.append(g + s.adjoint_gradient(dis))
    for a, b in zip(*out):
        assert rel_l2(a, b) < (1e-11 if precision == "fp64" else 1e-4)
