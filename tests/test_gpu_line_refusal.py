"""Meshes that the line operator serves or refuses, and the reason it gives."""
import dataclasses

import numpy as np
import pytest

from hirensi_b200.mesh import box_mesh
from problems import RHO, rel_l2, tiny

pytestmark = pytest.mark.gpu


def _solver(mesh, p):
    from hirensi_b200.solver import Solver
    rng = np.random.default_rng(4)
    mu = RHO * rng.uniform(200.0, 400.0, mesh.nj) ** 2
    s = Solver("fp64")
    s.set_mesh(mesh, RHO)
    s.assemble(2 * mu, mu)
    s.set_history(mesh.store_eq)
    src = mesh.equations(mesh.store_nodes[-5:-4], comps=(2,))
    s.set_shots(p["nstep"], p["dt"], src, np.eye(1), p["ftab"])
    s.set_receivers(src, mesh.store_position(src))
    return s


def _row_swapped(mesh, first, a, b):
    """Two equations of one node exchanged: DOFs a, b of the last node whose DOF `first` is free."""
    j = int(np.nonzero(mesh.ID[:, first] >= 0)[0][-1])
    ID = mesh.ID.copy()
    ID[j, [a, b]] = ID[j, [b, a]]
    return dataclasses.replace(mesh, ID=ID)


def _tilted(mesh):
    """The PML's outer nodes at x+ moved in y and z: its grid lines leave the axes."""
    xyz = mesh.xyz.copy()
    out = xyz[:, 0] > 0.5 * mesh.nx * mesh.h + 0.1 * mesh.h
    xyz[out, 1] += 0.1 * (xyz[out, 0] - 0.5 * mesh.nx * mesh.h)
    return dataclasses.replace(mesh, xyz=xyz)


@pytest.mark.parametrize("change,reason", [(lambda m: _row_swapped(m, 0, 0, 1), "displacement equations"),
                                           (lambda m: _row_swapped(m, 3, 4, 5), "stress equations"),
                                           (_tilted, "weights")])
def test_reason_of_a_refusal(gpu_lib, change, reason):
    from hirensi_b200.capi import HRN_EARG, HrnError
    p = tiny(nshot=1, nstep=10)
    with _solver(change(box_mesh(3, 2, 2, 2.5, 2)), p) as s:
        s.set_variant(96, 96)
        with pytest.raises(HrnError) as e:
            s.forward()
        assert e.value.code == HRN_EARG and reason in str(e.value)
        s.set_variant(0, 0)   # the tuner takes a variant that serves it
        s.forward()
        assert s.variant()[0] not in (96, 97, 98)


@pytest.mark.parametrize("h,shift", [(1.3, 0.0), (3.3, 0.0), (2.5, 1000.1), (2.5, 500000.3), (1.0 / 3.0, 7.7)])
def test_spacings_and_offsets_that_are_not_dyadic(gpu_lib, h, shift):
    """Aligned meshes whose coordinates carry rounding; bar as between any two FP64 variants."""
    p = tiny(nshot=1, nstep=20)
    mesh = box_mesh(5, 4, 3, h, 2)
    pml = mesh.pml_param.copy()
    pml[:4, 3] += shift
    mesh = dataclasses.replace(mesh, xyz=mesh.xyz + [shift, shift, 0.0], pml_param=pml)
    with _solver(mesh, p) as s:
        s.set_variant(96, 96)
        s.forward()
        a = s.history(0)
        s.set_variant(41, 41)
        s.forward()
        assert rel_l2(a, s.history(0)) < 1e-11
