"""History, source and receiver lists that are refused: nothing of them is in force
afterwards, a solve says what is missing, and setting the list again completes the problem."""
import numpy as np
import pytest

from problems import RHO, tiny

pytestmark = pytest.mark.gpu


def _lists(s, p, bad=None):
    """The three setters, or those up to `bad`, which is given an equation out of range."""
    from hirensi_b200.capi import HrnError
    far = np.int32(p["mesh"].neq + 100000)
    calls = dict(history=lambda e: s.set_history(np.append(p["mesh"].store_eq, e).astype(np.int32)),
                 shots=lambda e: s.set_shots(p["nstep"], p["dt"], np.append(p["src_eq"], e).astype(np.int32),
                                             np.vstack([p["src_b"]] + [p["src_b"][:1]] * e.size), p["ftab"]),
                 receivers=lambda e: s.set_receivers(np.append(p["eqdis"], e).astype(np.int32),
                                                     np.append(p["eqdis_map"], np.zeros(e.size, np.int32)).astype(np.int32)))
    for name, call in calls.items():
        if name == bad:
            with pytest.raises(HrnError):
                call(np.full(50000, far, np.int32) if name != "shots" else np.array([far], np.int32))
            return
        else:
            call(np.zeros(0, np.int32))


def _solve(s):
    s.set_variant(96, 96)
    s.forward()
    return s.traces()


@pytest.mark.parametrize("ckpt", [0, 7])
@pytest.mark.parametrize("bad", ["history", "shots", "receivers"])
def test_refused_list_is_dropped(gpu_lib, bad, ckpt):
    from hirensi_b200.capi import HrnError
    from hirensi_b200.solver import Solver
    p = tiny(nshot=2, nstep=20)
    with Solver("fp64") as s:
        s.set_mesh(p["mesh"], RHO)
        s.assemble(p["lam"], p["mu"])
        _lists(s, p)
        s.set_checkpointing(ckpt)
        ref = _solve(s)
        _lists(s, p)
        _lists(s, p, bad)
        if bad == "receivers":
            assert _solve(s).size == 0 and s.misfit(np.zeros((2, 0, p["nstep"] + 1))) == 0.0
        else:
            with pytest.raises(HrnError):
                s.forward()
        _lists(s, p)
        assert np.array_equal(_solve(s), ref)


def test_time_functions_that_are_not_finite(gpu_lib):
    from hirensi_b200.capi import HrnError
    from hirensi_b200.solver import Solver
    p = tiny(nshot=2, nstep=20)
    with Solver("fp64") as s:
        s.set_mesh(p["mesh"], RHO)
        s.assemble(p["lam"], p["mu"])
        _lists(s, p)
        ref = _solve(s)
        f = np.repeat(p["ftab"], 2, axis=1)
        f[0, 3, 1] = np.nan
        with pytest.raises(HrnError):
            s.set_shots(2 * p["nstep"] + 1, p["dt"], p["src_eq"], p["src_b"], f)
        for call in (s.forward, lambda: s.history(0)):
            with pytest.raises(HrnError):
                call()
        _lists(s, p)
        assert np.array_equal(_solve(s), ref)


def test_refused_when_the_operator_comes(gpu_lib):
    """Lists set before the operator are looked at when it comes; the good ones stay."""
    from hirensi_b200.capi import HrnError
    from hirensi_b200.solver import Solver
    p = tiny(nshot=1, nstep=10)
    store = p["mesh"].store_eq
    with Solver("fp64") as s, Solver("fp64") as r:
        for x, h in ((s, np.append(store, p["mesh"].neq).astype(np.int32)), (r, store)):
            x.set_history(h)
            x.set_shots(p["nstep"], p["dt"], p["src_eq"], p["src_b"], p["ftab"])
            x.set_mesh(p["mesh"], RHO)
        with pytest.raises(HrnError):
            s.assemble(p["lam"], p["mu"])
        with pytest.raises(HrnError):
            s.forward()
        r.assemble(p["lam"], p["mu"])
        s.set_history(store)
        for x in (s, r):
            x.set_receivers(p["eqdis"], p["eqdis_map"])
            x.set_variant(41, 41)
            x.forward()
        assert np.array_equal(s.history(0), r.history(0))


def test_receivers_set_after_the_data_or_a_checkpointed_forward(gpu_lib):
    """Data and traces are those of the receivers they came with: a longer list reads past neither."""
    from hirensi_b200.capi import HrnError
    from hirensi_b200.solver import Solver
    p = tiny(nshot=1, nstep=20)
    mesh = p["mesh"]
    some, every = (p["eqdis"][:3], p["eqdis_map"][:3]), (p["eqdis"], p["eqdis_map"])
    zero = np.zeros((1, len(p["eqdis"]), p["nstep"] + 1))
    with Solver("fp64") as s:
        s.set_mesh(mesh, RHO)
        s.assemble(p["lam"], p["mu"])
        s.set_history(mesh.store_eq)
        s.set_shots(p["nstep"], p["dt"], p["src_eq"], p["src_b"], p["ftab"])
        s.set_receivers(*some)
        s.set_data(zero[:, :3])
        s.set_variant(41, 41)
        s.forward()
        few = s.traces()
        s.set_receivers(*every)             # the whole history: traces of any receivers
        assert np.array_equal(s.traces()[:, :3], few)
        for call in (lambda: s.misfit(None), lambda: s.adjoint_gradient(None)):
            with pytest.raises(HrnError):
                call()
        assert s.misfit(zero) > 0.0
        s.set_checkpointing(5)
        s.forward()
        s.set_receivers(*every)             # the same list changes nothing
        assert np.array_equal(s.traces()[:, :3], few)
        s.set_receivers(*some)
        with pytest.raises(HrnError):
            s.traces()
        s.forward()
        s.set_receivers(*every)
        for call in (s.traces, lambda: s.misfit(zero), lambda: s.adjoint_gradient(zero)):
            with pytest.raises(HrnError):
                call()
