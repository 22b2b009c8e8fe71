"""time_stage times stages alone: the line operator's preparation belongs to the warm-up step."""
import pytest

from problems import RHO, tiny

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adjoint", [False, True])
def test_preparation_is_not_timed(gpu_lib, adjoint):
    from hirensi_b200.solver import Solver
    p = tiny(nshot=2, nstep=5)
    with Solver("fp64") as s:
        s.set_mesh(p["mesh"], RHO)
        s.assemble(p["lam"], p["mu"])
        s.set_history(p["mesh"].store_eq)
        s.set_shots(p["nstep"], p["dt"], p["src_eq"], p["src_b"], p["ftab"])
        s.set_receivers(p["eqdis"], p["eqdis_map"])
        s.set_variant(97, 97)
        s.forward()
        n = []
        for steps in (1, 2, 3):
            before = s.launch_count()
            assert s.time_stage(adjoint, steps) > 0.0
            n.append(s.launch_count() - before)
    step = n[2] - n[1]
    assert n[1] - n[0] == step == 8                 # two launches a stage
    assert n[0] == 2 * step + 2                     # warm-up and one step; P and Z formed once
