"""Line-operator stage variants (96, 97, 98: up to 1, 2, 4 shots per thread) against the
FP64 oracle, and against the row-parallel kernel on the assembled operator.

Bars as for the other matrix-free variants: relative L2 1e-10 in FP64, 1e-4 (histories)
and 1e-3 (gradients) in FP32 stepping against the oracle; 1e-11 between two FP64 variants
of the same steps (their sums differ in order only)."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from problems import RHO, oracle_forward, rel_l2, tiny, traces_from_history

pytestmark = pytest.mark.gpu


def _solver(p, precision="fp64", mesh=None):
    from hirensi_b200.solver import Solver
    s = Solver(precision)
    m = mesh or p["mesh"]
    s.set_mesh(m, RHO)
    s.assemble(p["lam"], p["mu"])
    s.set_history(m.store_eq)
    s.set_shots(p["nstep"], p["dt"], p["src_eq"], p["src_b"], p["ftab"])
    s.set_receivers(p["eqdis"], p["eqdis_map"])
    return s


def _data(p, seed=3):
    rng = np.random.default_rng(seed)
    return 1e-6 * rng.standard_normal((p["nshot"], len(p["eqdis"]), p["nstep"] + 1))


def _run(p, variant, precision="fp64", ckpt=0, lambda_2mu=False, mesh=None, fwd=None):
    with _solver(p, precision, mesh) as s:
        s.set_variant(fwd or variant, variant)
        if ckpt:
            s.set_checkpointing(ckpt)
        s.forward()
        hist = None if ckpt else [s.history(k) for k in range(p["nshot"])]
        tr = s.traces()
        J = s.misfit(_data(p))
        g = s.adjoint_gradient(_data(p), lambda_2mu=lambda_2mu, keep_p=True)
        ph = s.adjoint_history(p["nshot"] - 1)
    return hist, tr, J, g, ph


def _same(a, b, tol=1e-11):
    if a[0] is not None and b[0] is not None:
        for x, y in zip(a[0], b[0]):
            assert rel_l2(x, y) < tol
    assert rel_l2(a[1], b[1]) < tol
    assert abs(a[2] - b[2]) <= tol * abs(b[2])
    assert rel_l2(a[3][0], b[3][0]) < tol and rel_l2(a[3][1], b[3][1]) < tol
    assert rel_l2(a[4], b[4]) < tol


@pytest.mark.parametrize("precision,variant,nshot", [("fp64", 96, 1), ("fp64", 97, 2), ("fp32", 98, 4), ("fp32", 96, 3)])
def test_line_operator_matches_oracle(gpu_lib, precision, variant, nshot):
    p = tiny(nshot=nshot, nstep=120)
    om, S, hist = oracle_forward(p, p["lam"], p["mu"])
    dis = np.stack([0.5 * traces_from_history(p, h) for h in hist])
    bar_u, bar_g = (1e-10, 1e-10) if precision == "fp64" else (1e-4, 1e-3)
    with _solver(p, precision) as s:
        s.set_variant(variant, variant)
        s.forward()
        for k in range(nshot):
            assert rel_l2(s.history(k), hist[k]) < bar_u
        s.misfit(dis)
        gl, gm = s.adjoint_gradient(dis)
        assert s.variant() == (variant, variant)
    rl, rm = np.zeros_like(gl), np.zeros_like(gm)
    for k in range(nshot):
        pk = S.adjoint(p["nstep"], p["dt"], p["mesh"].store_eq, hist[k], p["eqdis"], p["eqdis_map"], dis[k])
        a, b = O.control(om, p["nstep"], p["dt"], p["mesh"].store_eq, hist[k], pk)
        rl += a
        rm += b
    assert rel_l2(gl, rl) < bar_g and rel_l2(gm, rm) < bar_g


@pytest.mark.parametrize("shape,nshot,variant", [
    ((1, 1, 1, 1), 1, 96), ((3, 1, 2, 1), 2, 97), ((2, 5, 3, 2), 3, 98), ((5, 4, 2, 3), 4, 97), ((3, 3, 2, 1), 5, 96),
    ((3, 2, 1, 2), 6, 97), ((2, 3, 2, 1), 7, 97), ((4, 3, 2, 1), 8, 97), ((4, 3, 2, 1), 8, 96)])
def test_line_operator_equals_assembled_operator(gpu_lib, shape, nshot, variant):
    nx, ny, nz, npml = shape
    p = tiny(nshot=1, nstep=24)
    from hirensi_b200.mesh import box_mesh
    mesh = box_mesh(nx, ny, nz, 2.5, npml)
    rng = np.random.default_rng(7)
    mu = RHO * rng.uniform(200.0, 400.0, mesh.nj) ** 2
    surf = mesh.store_nodes[np.abs(mesh.xyz[mesh.store_nodes, 2]) < 1e-9]
    src = mesh.equations(rng.choice(surf, nshot, replace=False), comps=(2,))
    rec = mesh.equations(surf[:5])
    p.update(mesh=mesh, lam=2 * mu, mu=mu, nshot=nshot, src_eq=src, src_b=np.eye(nshot),
             ftab=np.stack([p["ftab"][0]] * nshot), eqdis=rec, eqdis_map=mesh.store_position(rec))
    _same(_run(p, variant), _run(p, 41))
    _same(_run(p, variant, lambda_2mu=True), _run(p, 41, lambda_2mu=True))


def _distorted(mesh, seed=1):
    """The nodes inside the regular domain moved off the lattice (the PML stays aligned)."""
    rng = np.random.default_rng(seed)
    inner = mesh.node_mat_id == 0
    xyz = mesh.xyz.copy()
    d = 0.02 * mesh.h * rng.uniform(-1.0, 1.0, xyz.shape)
    d[np.abs(xyz[:, 2]) < 1e-9, 2] = 0.0
    xyz[inner] += d[inner]
    return dataclasses.replace(mesh, xyz=xyz)


@pytest.mark.parametrize("variant,nshot", [(96, 3), (97, 4)])
def test_distorted_regular_domain(gpu_lib, variant, nshot):
    p = tiny(nshot=nshot, nstep=30)
    mesh = _distorted(p["mesh"])
    _same(_run(p, variant, mesh=mesh), _run(p, 41, mesh=mesh))


@pytest.mark.parametrize("ckpt", [1, 7, 30])
@pytest.mark.parametrize("fwd", [97, 41])
def test_checkpoints_and_mixed_variants(gpu_lib, ckpt, fwd):
    """Checkpoints hold the states in the order of the variant that wrote them."""
    p = tiny(nshot=2, nstep=30)
    full = _run(p, 41)
    _same(_run(p, 97, ckpt=ckpt, fwd=fwd), full)
    _same(_run(p, 41, ckpt=ckpt, fwd=fwd), full)
    with _solver(p) as s, _solver(p) as r:
        s.set_variant(fwd, fwd)
        r.set_variant(41, 41)
        for x in (s, r):
            x.set_checkpointing(ckpt)
            x.forward()
        at = (p["nstep"] // ckpt) * ckpt
        for a, b in zip(s.state(at, 1), r.state(at, 1)):
            assert rel_l2(a, b) < 1e-11
        # another variant chosen after the forward: the segments are recomputed as they were stepped
        s.set_variant(41 if fwd == 97 else 97, 41)
        g, h = s.adjoint_gradient(_data(p)), r.adjoint_gradient(_data(p))
        assert rel_l2(g[0], h[0]) < 1e-11 and rel_l2(g[1], h[1]) < 1e-11


def test_sources_and_history_on_stress_rows(gpu_lib):
    """Loads on stress equations reach them (no ordinary set-up has any)."""
    p = tiny(nshot=2, nstep=30)
    mesh = p["mesh"]
    stress = int(mesh.ID[np.nonzero(mesh.node_mat_id == 1)[0][3], 4])
    p["src_eq"] = np.array([p["src_eq"][0], stress], dtype=np.int32)
    p["src_b"] = np.array([[1.0, 0.0], [0.0, 1e-3]])
    _same(_run(p, 97), _run(p, 41))


def test_unsuited_numbering_takes_another_variant(gpu_lib):
    """A node whose displacement equations are not in a row: the line variants refuse it,
    and the tuner picks one that serves it."""
    from hirensi_b200.capi import HrnError
    p = tiny(nshot=1, nstep=20)
    mesh = p["mesh"]
    j = int(np.nonzero(mesh.node_mat_id == 2)[0][-1])
    while mesh.ID[j, 0] < 0:
        j -= 1
    ID = mesh.ID.copy()
    ID[j, [0, 1]] = ID[j, [1, 0]]
    odd = dataclasses.replace(mesh, ID=ID)
    with _solver(p, mesh=odd) as s:
        s.set_variant(96, 96)
        with pytest.raises(HrnError):
            s.forward()
        s.set_variant(0, 0)
        s.forward()
        assert s.variant()[0] not in (96, 97, 98)
        ref = s.traces()
    with _solver(p) as s:
        s.set_variant(41, 41)
        s.forward()
        assert rel_l2(ref, s.traces()) < 1e-11


def test_variant_survives_another_shot_count(gpu_lib):
    p = tiny(nshot=4, nstep=20)
    with _solver(p) as s:
        s.set_variant(97, 97)
        s.forward()
        s.set_shots(p["nstep"], p["dt"], p["src_eq"][:3], np.eye(3), p["ftab"][:3])
        s.forward()
        odd = s.traces()
    q = dict(p, nshot=3, src_eq=p["src_eq"][:3], src_b=np.eye(3), ftab=p["ftab"][:3])
    with _solver(q) as s:
        s.set_variant(41, 41)
        s.forward()
        assert rel_l2(odd, s.traces()) < 1e-11


@pytest.mark.parametrize("nshot,variant", [(8, 98), (7, 96)])
def test_register_elements_of_large_fp32_grids(gpu_lib, nshot, variant):
    """Enough elements and shots for the kernel that keeps an element in registers."""
    from hirensi_b200.configs import inversion_config
    from hirensi_b200.solver import Solver
    p = inversion_config(nstep=12, nx=21, ny=20, nz=18, npml=1, shots=tuple((2.5 * k - 10.0, 5.0) for k in range(nshot)),
                         receivers=(-10.0, 0.0, 10.0), fr=900.0)
    dis = 1e-6 * np.random.default_rng(2).standard_normal((nshot, len(p.eqdis), p.nstep + 1))
    out = {}
    for prec, v in (("fp32", variant), ("fp64", 41)):
        with Solver(prec) as s:
            s.set_mesh(p.mesh, RHO)
            s.assemble(p.lam_true, p.mu_true)
            s.set_history(p.mesh.store_eq)
            s.set_shots(p.nstep, p.dt, p.src_eq, p.src_b, p.ftab)
            s.set_receivers(p.eqdis, p.eqdis_map)
            s.set_variant(v, v)
            s.forward()
            s.misfit(dis)
            out[prec] = (s.history(nshot - 1), *s.adjoint_gradient(dis))
    for a, b, bar in zip(out["fp32"], out["fp64"], (1e-4, 1e-3, 1e-3)):
        assert rel_l2(a, b) < bar
