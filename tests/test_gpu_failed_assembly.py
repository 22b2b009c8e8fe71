"""A reassembly that fails leaves the operator before it in force, whichever variant steps."""
import numpy as np
import pytest

from problems import RHO, rel_l2, tiny

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [96, 90, 41])
def test_forward_after_a_failed_reassembly(gpu_lib, variant):
    import torch
    from hirensi_b200.capi import HrnError
    from hirensi_b200.solver import Solver
    p = tiny(nshot=2, nstep=30)
    mesh = p["mesh"]
    bad = torch.from_numpy(p["lam"]).cuda()
    inner = int(np.nonzero(mesh.node_mat_id == 0)[0][0])
    bad[inner] = float("nan")   # entries outside the pattern of the first assembly
    mu = torch.from_numpy(p["mu"]).cuda()
    torch.cuda.synchronize()
    with Solver("fp64") as s:
        s.set_mesh(mesh, RHO)
        s.assemble(p["lam"], p["mu"])
        s.set_history(mesh.store_eq)
        s.set_shots(p["nstep"], p["dt"], p["src_eq"], p["src_b"], p["ftab"])
        s.set_receivers(p["eqdis"], p["eqdis_map"])
        s.set_variant(variant, variant)
        s.forward()
        ref = s.history(1)
        with pytest.raises(HrnError):
            s.assemble_device(bad.data_ptr(), mu.data_ptr())
        s.forward()
        assert rel_l2(s.history(1), ref) < 1e-11
        s.assemble(p["lam"], p["mu"])   # a good one restores every variant
        s.set_variant(variant, variant)
        s.forward()
        assert np.array_equal(s.history(1), ref)
