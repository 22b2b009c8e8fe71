"""The work that users of this framework have it do, as measurable cases.

Three kinds of calls carry it:

* solves (``evaluation``, ``forward``, ``csr_forward``): a model is assembled, the shots
  are stepped forward, and for an inversion the misfit, the adjoint and the gradient
  follow.  These are nearly all of a run's time.  Meshes from a few elements to a few
  hundred thousand, even and odd sizes, one to eight shots, FP64 and FP32 stepping, whole
  histories and checkpoints, even and uneven records, stored and matrix-free operators,
  and operators that the caller assembled;
* the model update between two solves (``update``): TV, norms, the coupled L-BFGS direction;
* layers of the learned preconditioner (``conv_forward``, ``conv_backward``).

Time steps are fewer than a production record's 2000-8000, which only repeat the same
step; the source frequency is raised to match, so that waves cross the model.

FP32 stepping keeps its wavefield in FP32, so seismograms and gradients of those solves
are returned in that type (exact for the seismograms).
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from hirensi_b200 import capi
from hirensi_b200.configs import RHO, extend_into_pml, time_table, vs_to_lame
from hirensi_b200.inversion import DeviceBackend
from hirensi_b200.mesh import GLL_TO_LOCAL, box_mesh
from hirensi_b200.solver import Solver

H, DT = 2.5, 1.0e-4


def _solve(name, kind, nx, ny, nz, npml, shots, nstep, precision, ckpt=0, uneven=False, matrix_free=False):
    return dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, npml=npml, shots=shots, nstep=nstep, precision=precision,
                ckpt=ckpt, uneven=uneven, matrix_free=matrix_free)


def listed():
    return [
        # a layer of the preconditioner on the inversion mesh's node lattice (17 x 33 x 33): the first, 6 inputs
        dict(name="conv_forward_17x33x33", kind="conv_forward", cin=6, cout=16, lz=17, ly=33, lx=33, relu=True),
        # a hidden layer's backward pass on the training mesh's lattice (41 x 81 x 81)
        dict(name="conv_backward_41x81x81", kind="conv_backward", cin=16, cout=16, lz=41, ly=81, lx=81, relu=True),
        # the model update of one inversion iteration on the inversion mesh, L-BFGS memory 5
        dict(name="update_16x16x8", kind="update", nx=16, ny=16, nz=8, npml=3, memory=5),
        # the smallest evaluation: a check of a set-up, a unit test, a gradient check
        _solve("evaluation_4x4x2_fp64", "evaluation", 4, 4, 2, 1, 1, 60, "fp64"),
        # the forward-only workload: one source, seismograms
        _solve("forward_16x16x8_fp64", "forward", 16, 16, 8, 3, 1, 300, "fp64"),
        # the plain inversion workload: 4 shots, FP64
        _solve("evaluation_16x16x8_fp64", "evaluation", 16, 16, 8, 3, 4, 200, "fp64"),
        # the same with FP32 stepping, as the accelerated inversion runs it
        _solve("evaluation_16x16x8_fp32", "evaluation", 16, 16, 8, 3, 4, 200, "fp32"),
        # an odd mesh and an odd number of shots with uneven records
        _solve("evaluation_11x7x5_fp64_uneven", "evaluation", 11, 7, 5, 2, 3, 150, "fp64", uneven=True),
        # the training mesh of the preconditioner, a full batch of 8 shots
        _solve("evaluation_40x40x20_fp32", "evaluation", 40, 40, 20, 3, 8, 60, "fp32"),
        # uneven shots with checkpoints, as large record sets are inverted
        _solve("evaluation_32x24x16_fp32_ckpt", "evaluation", 32, 24, 16, 4, 5, 100, "fp32", ckpt=25, uneven=True),
        # a large mesh whose operator is applied without storing it
        _solve("evaluation_64x64x32_fp32_mfree", "evaluation", 64, 64, 32, 4, 4, 24, "fp32", ckpt=12, matrix_free=True),
        # the drop-in boundary: matrices assembled by the caller, one source
        _solve("csr_forward_16x16x8_fp64", "csr_forward", 16, 16, 8, 3, 1, 200, "fp64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _equations(nx, ny, nz, npml):
    """About the number of equations of a box mesh: 3 per node, 9 inside the PML."""
    n = (2 * (nx + 2 * npml) + 1) * (2 * (ny + 2 * npml) + 1) * (2 * (nz + npml) + 1)
    r = (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1)
    return 9 * n - 6 * r


def draw(rng):
    kind = rng.choice(["evaluation"] * 8 + ["forward"] * 3 + ["update", "conv_forward", "conv_backward", "csr_forward"])
    if kind.startswith("conv"):
        lz, ly, lx = _log_int(rng, 5, 41), _log_int(rng, 9, 81), _log_int(rng, 9, 81)
        return dict(kind=kind, cin=rng.choice([4, 6, 16]), cout=rng.choice([2, 16]), lz=lz, ly=ly, lx=lx,
                    relu=rng.random() < 0.75)
    if kind == "update":
        return dict(kind=kind, nx=_log_int(rng, 4, 32), ny=_log_int(rng, 4, 32), nz=_log_int(rng, 2, 16),
                    npml=rng.randint(1, 4), memory=rng.randint(1, 15))
    big = kind != "csr_forward"
    nx = _log_int(rng, 3, 40 if big else 16)
    ny = max(2, min(40 if big else 16, round(nx * rng.uniform(0.6, 1.4))))
    nz = max(2, min(20 if big else 8, round(nx * rng.uniform(0.35, 0.7))))
    npml = rng.randint(1, 4)
    shots = 1 if kind == "csr_forward" else rng.randint(1, 8)
    precision = rng.choice(["fp64", "fp32"])
    # a pass of at most about 4e9 equation-shot-steps, as the largest listed one
    cap = 4.0e8 / (_equations(nx, ny, nz, npml) * shots)
    nstep = max(8, min(_log_int(rng, 20, 300), int(cap)))
    uneven = kind == "evaluation" and shots > 1 and rng.random() < 0.3
    ckpt = rng.randint(5, 40) if kind == "evaluation" and rng.random() < 0.3 else 0
    free = kind == "evaluation" and rng.random() < 0.2
    c = _solve("", kind, nx, ny, nz, npml, shots, nstep, precision, ckpt, uneven, free)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs

@functools.lru_cache(maxsize=3)
def _mesh(nx, ny, nz, npml):
    return box_mesh(nx, ny, nz, H, npml)


def _model(case, mesh, rng):
    """Nodal (lambda, mu): Vs growing with depth, a random smooth anomaly, extended into the PML."""
    depth = case["nz"] * H
    z = np.clip(mesh.xyz[:, 2], -depth, 0.0)
    vs = rng.uniform(180.0, 220.0) + rng.uniform(180.0, 220.0) * (-z / depth)
    half = 0.5 * np.array([case["nx"], case["ny"]]) * H
    at = np.array([rng.uniform(-0.5, 0.5) * half[0], rng.uniform(-0.5, 0.5) * half[1], -rng.uniform(0.2, 0.7) * depth])
    d2 = ((mesh.xyz - at) ** 2).sum(axis=1)
    vs = vs * (1.0 + rng.uniform(0.2, 0.4) * rng.choice([-1.0, 1.0]) * np.exp(-d2 / (0.25 * depth) ** 2))
    return vs_to_lame(extend_into_pml(mesh, vs))


def _survey(case, seed):
    """Mesh, model, sources, receivers, per-shot records and measured data of a case."""
    rng = np.random.default_rng(seed)
    mesh = _mesh(case["nx"], case["ny"], case["nz"], case["npml"])
    lam, mu = _model(case, mesh, rng)
    S, N = case["shots"], case["nstep"]
    NX, NY, NZ = mesh.lattice
    p = 2 * case["npml"]
    ii, jj = np.meshgrid(np.arange(p + 1, NX - p - 1), np.arange(p + 1, NY - p - 1))
    surface = (ii + NX * (jj + NY * (NZ - 1))).ravel()
    src_nodes = rng.choice(surface, size=S, replace=False)
    src_eq = mesh.equations(src_nodes, comps=(2,))
    fr = 1.6 / (N * DT)                     # a record spans about 1.6 periods of the source
    ftab = np.stack([time_table(N, DT, 2, fr * f) for f in rng.uniform(0.8, 1.2, S)])
    nrec = min(25, surface.size)
    rec = np.sort(rng.choice(surface, size=nrec, replace=False))
    eqdis = mesh.equations(rec)
    lengths, mask = None, None
    if case["uneven"]:
        lengths = np.maximum(2, np.round(N * rng.uniform(0.6, 1.0, S))).astype(np.int32)
        lengths[rng.integers(S)] = N
        mask = np.repeat(rng.random((S, nrec)) < 0.7, 3, axis=1).astype(np.uint8)
        mask[:, :3] = 1
    # measured records: the far field of a vertical force, delayed by the distance, with 5 % noise
    r = np.maximum(np.linalg.norm(mesh.xyz[rec][None] - mesh.xyz[src_nodes][:, None], axis=2), 0.5 * H)   # [S, nrec]
    vs = np.sqrt(mu / RHO)[rec].mean()
    amp = 1.0 / (4.0 * math.pi * RHO * vs * vs * r)
    t = np.arange(N + 1)[None, None, :] - np.round(r / (vs * DT)).astype(int)[:, :, None]
    pulse = np.take_along_axis(np.broadcast_to(ftab[:, None, :, 0], t.shape), np.clip(t, 0, N), axis=2) * (t > 0)
    wave = amp[:, :, None] * pulse
    dis = np.stack([0.3 * wave, 0.2 * wave, wave], axis=2).reshape(S, 3 * nrec, N + 1)
    dis = dis * (1.0 + 0.05 * rng.standard_normal(dis.shape))
    return dict(mesh=mesh, lam=lam, mu=mu, src_eq=src_eq, src_b=np.eye(S), ftab=ftab, eqdis=eqdis,
                eqdis_map=mesh.store_position(eqdis), lengths=lengths, mask=mask, dis=np.ascontiguousarray(dis))


def _solver(case, p):
    s = Solver(case["precision"])
    s.set_mesh(p["mesh"], RHO)
    if case["matrix_free"]:
        s.set_operator_mode(True)
    s.set_history(p["mesh"].store_eq)
    return s


def _problem(case, s, p):
    s.set_shots(case["nstep"], DT, p["src_eq"], p["src_b"], p["ftab"])
    s.set_receivers(p["eqdis"], p["eqdis_map"])
    if p["lengths"] is not None:
        s.set_shot_records(p["lengths"], p["mask"])
    if case["ckpt"]:
        s.set_checkpointing(case["ckpt"])
    s.set_data(p["dis"])


def _smooth(gen, n):
    """A nodal vector of unit scale with some structure."""
    x = torch.linspace(0.0, 12.0, n, dtype=torch.float64, device="cuda")
    a = torch.rand(4, generator=gen, dtype=torch.float64).tolist()
    return torch.sin(x * (1 + a[0]) + 6 * a[1]) + 0.3 * torch.cos(x * (5 + a[2]) + 6 * a[3])


def _update_inputs(case, seed):
    """Models and gradients of the last memory + 2 iterates, restricted to the regular domain."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator().manual_seed(seed)
    mesh = _mesh(case["nx"], case["ny"], case["nz"], case["npml"])
    n = mesh.nj
    lam, mu = _model(dict(case), mesh, rng)
    keep = torch.from_numpy((mesh.node_mat_id <= 1).astype(np.float64)).cuda()
    m, g = [], []
    cur = [torch.from_numpy(lam).cuda(), torch.from_numpy(mu).cuda()]
    grad = [0.02 * _smooth(gen, n), 0.05 * _smooth(gen, n)]
    for _ in range(case["memory"] + 2):
        m.append([v.clone() for v in cur])
        g.append([v.clone() for v in grad])
        step = [0.5 * _smooth(gen, n), 0.4 * _smooth(gen, n)]
        cur = [c + s for c, s in zip(cur, step)]
        grad = [gr + 0.02 * s + 0.002 * _smooth(gen, n) for gr, s in zip(grad, step)]
    return mesh, keep, m, g


def _conv_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    V, ci, co = case["lz"] * case["ly"] * case["lx"], case["cin"], case["cout"]
    x = torch.zeros(V, 16, device="cuda")
    x[:, :ci] = torch.randn(V, ci, generator=gen, device="cuda").relu_()
    w = torch.randn(co, ci, 27, generator=gen, device="cuda") * math.sqrt(2.0 / (27 * ci))
    b = 0.1 * torch.randn(co, generator=gen, device="cuda")
    gy = torch.zeros(V, 16, device="cuda")
    gy[:, :co] = torch.randn(V, co, generator=gen, device="cuda")
    return x.bfloat16(), w.bfloat16(), b, gy


def prepare(case, seed):
    kind = case["kind"]
    if kind.startswith("conv"):
        x, w, b, gy = _conv_inputs(case, seed)
        st = dict(case=case, L=capi.load(), x=x, w=w, b=b, gy=gy, y=torch.zeros_like(x),
                  stream=torch.cuda.current_stream().cuda_stream)
        if kind == "conv_backward":
            st["gx"] = torch.zeros(x.shape, device="cuda")
            st["gw"] = torch.zeros(w.shape, device="cuda")
            st["gb"] = torch.zeros_like(b)
            _conv_forward(st)
        return st
    if kind == "update":
        mesh, keep, m, g = _update_inputs(case, seed)
        s = Solver("fp64")
        s.set_mesh(mesh, RHO)
        back = DeviceBackend(s, mesh)
        torch.cuda.synchronize()
        img, _ = back.gradient_mass_inverse()
        back.lbfgs_setup(case["memory"], keep)
        out = [back.zeros() for _ in range(6)]
        for k in range(1, case["memory"] + 1):      # the pairs of the earlier iterations
            back.lbfgs_direction(k + 1, 1, *g[k], *g[k - 1], *m[k], *m[k - 1], *out[:2])
        torch.cuda.synchronize()
        return dict(case=case, s=s, back=back, m=m, g=g, img=img, out=out)
    p = _survey(case, seed)
    if kind == "csr_forward":
        with _solver(case, p) as s0:
            s0.assemble(p["lam"], p["mu"])
            mats, dm = [s0.operator_csr(k) for k in range(3)], s0.diag_m()
        s = Solver(case["precision"])
        s.set_operator_csr(*mats, dm)
        s.set_history(p["mesh"].store_eq)
        _problem(case, s, p)
        return dict(case=case, s=s)
    s = _solver(case, p)
    lam, mu = torch.from_numpy(p["lam"]).cuda(), torch.from_numpy(p["mu"]).cuda()
    torch.cuda.synchronize()
    s.assemble_device(lam.data_ptr(), mu.data_ptr())     # fixes the sparsity pattern
    _problem(case, s, p)
    return dict(case=case, s=s, lam=lam, mu=mu)


# ---------------------------------------------------------------------------
# one pass

def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _ok(rc):
    if rc:
        raise RuntimeError(f"hirensi_b200 error {rc}")


def _conv_forward(st):
    c = st["case"]
    _ok(st["L"].hrn_cnn_conv3d_forward(c["cin"], c["cout"], c["lz"], c["ly"], c["lx"], _ptr(st["x"]), _ptr(st["w"]),
                                       _ptr(st["b"]), int(c["relu"]), _ptr(st["y"]), C.c_void_p(st["stream"])))
    return st["y"]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "conv_forward":
        return _conv_forward(state)
    if kind == "conv_backward":
        c = case
        _ok(state["L"].hrn_cnn_conv3d_backward(c["cin"], c["cout"], c["lz"], c["ly"], c["lx"], _ptr(state["x"]),
                                               _ptr(state["w"]), _ptr(state["y"]), int(c["relu"]), _ptr(state["gy"]),
                                               _ptr(state["gx"]), _ptr(state["gw"]), _ptr(state["gb"]),
                                               C.c_void_p(state["stream"])))
        return state["gx"], state["gw"], state["gb"]
    if kind == "update":
        # the iteration's model update: TV with its adaptive factor, gradient-mass scaling, direction, step cap
        b, (m0, m1), (g0, g1) = state["back"], state["m"][-2:], state["g"][-2:]
        p_l, p_m, reg_l, reg_m, s_l, s_m = state["out"]
        cost_l, cost_m = b.tv(*m1, reg_l, reg_m)
        f_l, f_m = 0.3 * b.norm2(g1[0]) / b.norm2(reg_l), 0.3 * b.norm2(g1[1]) / b.norm2(reg_m)
        b.axpby(1.0, g1[0], f_l, reg_l, s_l)
        b.axpby(1.0, g1[1], f_m, reg_m, s_m)
        b.mul(s_l, state["img"], s_l)
        b.mul(s_m, state["img"], s_m)
        b.lbfgs_direction(case["memory"] + 2, 1, *g1, *g0, *m1, *m0, p_l, p_m)
        slope = b.dot(s_l, p_l) + b.dot(s_m, p_m)
        return dict(p_l=p_l, p_m=p_m, s_l=s_l, s_m=s_m, cost_l=cost_l, cost_m=cost_m, slope=slope,
                    cap_l=b.norminf(p_l), cap_m=b.norminf(p_m))
    s = state["s"]
    real = np.float32 if case["precision"] == "fp32" else np.float64
    if kind != "csr_forward":
        s.assemble_device(state["lam"].data_ptr(), state["mu"].data_ptr())
    s.forward()
    if kind != "evaluation":
        return s.traces().astype(real, copy=False)
    J = s.misfit()
    g_l, g_m = s.adjoint_gradient()
    return dict(misfit=J, g_lambda=g_l.astype(real, copy=False), g_mu=g_m.astype(real, copy=False))


# ---------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind.startswith("conv"):
        V, ci, co = case["lz"] * case["ly"] * case["lx"], case["cin"], case["cout"]
        f = 2.0 * 27 * ci * co * V
        if kind == "conv_forward":
            return dict(bytes=V * 2.0 * (ci + 16) + 54 * ci * co + 4 * co, flops=f)
        return dict(bytes=V * (2.0 * ci + 6.0 * co + 64.0) + 162.0 * ci * co + 4 * co, flops=2 * f)
    nx, ny, nz, npml = case["nx"], case["ny"], case["nz"], case["npml"]
    n = (2 * (nx + 2 * npml) + 1) * (2 * (ny + 2 * npml) + 1) * (2 * (nz + npml) + 1)
    r = (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1)
    if kind == "update":
        m = case["memory"]
        # gradients and models of two iterates, the pairs, the mass scaling; p and the scaled gradient out
        return dict(bytes=8.0 * n * (8 + 4 * m + 1 + 4), flops=n * (16.0 * m + 40) + 27 * nx * ny * nz * 120.0)
    S, N, b = case["shots"], case["nstep"], 8.0 if case["precision"] == "fp64" else 4.0
    neq = 9.0 * n - 6.0 * r
    # a step reads and writes the three state vectors; a history row is written, and read by the gradient.
    # A stage is about 400 operations per PML node and 780 per regular-domain node and shot.
    step_b, hist = 6 * neq * S * b, 3.0 * r * S * b
    stage_f = (400.0 * (n - r) + 780.0 * r) * S
    passes = 2 if kind == "evaluation" else 1
    hist_n = passes if kind == "evaluation" and not case["ckpt"] else 0
    model = 16.0 * n + (8.0 * 2 * n if kind == "evaluation" else 0.0) + 8.0 * S * 75 * (N + 1)
    return dict(bytes=passes * N * step_b + hist_n * N * hist + model, flops=passes * N * 4 * stage_f)


# ---------------------------------------------------------------------------
# the same results in 64 bits, from the element formulas, in torch

_D = torch.tensor([[-1.5, 2.0, -0.5], [-0.5, 0.0, 0.5], [0.5, -2.0, 1.5]], dtype=torch.float64)


class _Exact:
    """Elastic box mesh with its PML in 64 bits: fields are [nj, 9, S] (3 displacements, 6
    stresses), zero at constrained unknowns.  Points of an element run x fastest; every
    element is a cube of edge H, so a point's weight is w_a w_b w_c (H/2)^3."""

    def __init__(self, mesh, lam, mu):
        dev = "cuda"
        f64 = functools.partial(torch.as_tensor, dtype=torch.float64, device=dev)
        self.nj = mesh.nj
        eye, D = torch.eye(3, dtype=torch.float64), _D * (2.0 / H)
        self.G = torch.stack([torch.kron(eye, torch.kron(eye, D)), torch.kron(eye, torch.kron(D, eye)),
                              torch.kron(D, torch.kron(eye, eye))]).to(dev)       # d/dx, d/dy, d/dz at the 27 points
        w = f64([1 / 3, 4 / 3, 1 / 3])
        self.w = (w[:, None, None] * w[None, :, None] * w[None, None, :]).reshape(27) * (H / 2) ** 3
        pts = torch.as_tensor(mesh.inod[:, GLL_TO_LOCAL].astype(np.int64), device=dev)
        kind = torch.as_tensor(mesh.mtel, device=dev)
        self.rd, self.pml = pts[kind == 1], pts[kind == 2]
        self.lam, self.mu = f64(lam), f64(mu)
        self.free = torch.as_tensor(mesh.ID >= 0, device=dev).double()[:, :, None]
        # stretching: alpha, beta of the three axes at every node
        x, P = f64(mesh.xyz), mesh.pml_param
        al, be = torch.ones(mesh.nj, 3, dtype=torch.float64, device=dev), torch.zeros(mesh.nj, 3, dtype=torch.float64, device=dev)
        for row, ax, sign in ((0, 0, 1.0), (1, 0, -1.0), (2, 1, 1.0), (3, 1, -1.0), (5, 2, -1.0)):
            d = torch.clamp((x[:, ax] - P[row, 3]) * sign / P[row, 2], min=0.0) ** 2
            al[:, ax] += P[row, 0] * d
            be[:, ax] += P[row, 1] * d
        a, b = al.T, be.T
        o = ((1, 2), (0, 2), (0, 1))
        # weights of a derivative along axis k in C, K, G, and the mass factors a, b, c, d
        self.wt = [torch.stack([a[i] * a[j] for i, j in o]), torch.stack([a[i] * b[j] + a[j] * b[i] for i, j in o]),
                   torch.stack([b[i] * b[j] for i, j in o])]
        self.f = [a[0] * a[1] * a[2], a[0] * a[1] * b[2] + a[0] * a[2] * b[1] + a[1] * a[2] * b[0],
                  a[0] * b[1] * b[2] + a[1] * b[0] * b[2] + a[2] * b[0] * b[1], b[0] * b[1] * b[2]]
        self.two = f64([1, 1, 1, 2, 2, 2])[None, :, None]
        wr = self._add(self.rd, self.w[None, :].expand(len(self.rd), 27).reshape(-1, 1))[:, 0]
        self.wp = self._add(self.pml, self.w[None, :].expand(len(self.pml), 27).reshape(-1, 1))[:, 0]
        M = torch.zeros(mesh.nj, 9, 1, dtype=torch.float64, device=dev)
        M[:, :3, 0] = (RHO * (wr + self.wp * self.f[0]))[:, None]
        M[:, 3:] = (self.wp * self.f[0])[:, None, None] * self.two
        self.im = torch.where(self.free > 0, 1.0 / torch.where(M > 0, M, torch.ones_like(M)), torch.zeros_like(M))

    def _add(self, pts, v):
        return torch.zeros((self.nj,) + v.shape[1:], dtype=torch.float64, device="cuda").index_add_(0, pts.reshape(-1), v)

    def _grad(self, pts, u):
        """[3 axes][elements, 27, 3, S] derivatives of a displacement field at the points."""
        e = u[pts].flatten(2)
        return [torch.matmul(self.G[k], e).view(pts.shape + u.shape[1:]) for k in range(3)]

    def _div(self, pts, flux):
        """Adjoint of the gradient: node sums of sum_k dN/dx_k flux_k w."""
        w = self.w[None, :, None]
        s = sum(torch.matmul(self.G[k].T, flux[k].flatten(2) * w) for k in range(3))
        return self._add(pts, s.view((-1,) + flux[0].shape[2:]))

    SH = {(0, 1): 0, (0, 2): 1, (1, 2): 2}

    def _full(self, s):
        """[.., 3, 3, S] tensor of the six components xx, yy, zz, xy, xz, yz."""
        r = [[s[..., i, :] if i == j else s[..., 3 + self.SH[min(i, j), max(i, j)], :] for j in range(3)] for i in range(3)]
        return torch.stack([torch.stack(v, dim=-2) for v in r], dim=-3)

    def _elastic(self, t, shape):
        """lambda tr(t) I + 2 mu t of a tensor field given at nodes or points."""
        lam, mu = self.lam, self.mu
        if shape is not None:
            lam, mu = lam[shape], mu[shape]
        tr = t[..., 0, 0, :] + t[..., 1, 1, :] + t[..., 2, 2, :]
        eye = torch.eye(3, dtype=torch.float64, device="cuda")[:, :, None]
        return lam[..., None, None, None] * tr[..., None, None, :] * eye + 2 * mu[..., None, None, None] * t

    def apply(self, km, kt, h, adjoint):
        """-M^-1 (C km + K kt + G h), or the adjoint's: its transpose with C and G negated."""
        u = torch.zeros_like(km)
        g = torch.stack(self._grad(self.rd, kt[:, :3]), dim=-2)             # [e, 27, comp, axis, S]
        sig = self._elastic(0.5 * (g + g.transpose(-2, -3)), self.rd)
        u[:, :3] += self._div(self.rd, [sig[..., k, :] for k in range(3)])
        flux = 0.0
        for t, v in enumerate((km, kt, h)):
            sg = -1.0 if adjoint and t != 1 else 1.0
            wt = self.wt[t]                                                  # [axis, nj]
            s = self._full(v[:, 3:])
            s = sg * s if adjoint else -self._elastic(s, None)
            flux = flux + s * wt.T[:, None, :, None]                         # [nj, comp, axis, S]
            u[:, :3] += sg * (RHO * self.f[t + 1] * self.wp)[:, None, None] * v[:, :3]
            u[:, 3:] += sg * (self.f[t + 1] * self.wp)[:, None, None] * self.two * v[:, 3:]
            ge = [a * self.w[None, :, None, None] for a in self._grad(self.pml, v[:, :3])]
            gn = torch.stack([self._add(self.pml, a.flatten(0, 1)) for a in ge], dim=-2) * wt.T[:, None, :, None]
            if adjoint:
                gn = -sg * self._elastic(gn, None)
                gn = 0.5 * (gn + gn.transpose(-2, -3))
            e = [gn[:, i, i] for i in range(3)]
            e += [gn[:, i, j] + gn[:, j, i] for i, j in self.SH]
            u[:, 3:] += torch.stack(e, dim=1)
        u[:, :3] += self._div(self.pml, [flux[:, :, k][self.pml] for k in range(3)])
        return -self.im * u * self.free

    def step(self, x, src, dt, adjoint):
        """One RK4 step of (x1, x2, x3)' = (x2, x3, C x3 + K x2 + G x1 + src)."""
        x1, x2, x3 = x
        c = 0.5 * dt
        k1 = src[0] + self.apply(x3, x2, x1, adjoint)
        m2, t2, h2 = x3 + c * k1, x2 + c * x3, x1 + c * x2
        k2 = src[1] + self.apply(m2, t2, h2, adjoint)
        m3, t3, h3 = x3 + c * k2, x2 + c * m2, x1 + c * t2
        k3 = src[2] + self.apply(m3, t3, h3, adjoint)
        m4, t4, h4 = x3 + dt * k3, x2 + dt * m3, x1 + dt * t3
        k4 = src[3] + self.apply(m4, t4, h4, adjoint)
        d = dt / 6.0
        return (x1 + d * (x2 + 2 * t2 + 2 * t3 + t4), x2 + d * (x3 + 2 * m2 + 2 * m3 + m4), x3 + d * (k1 + 2 * k2 + 2 * k3 + k4))


def _exact_solve(case, seed):
    p = _survey(case, seed)
    mesh, S, N = p["mesh"], case["shots"], case["nstep"]
    E = _Exact(mesh, p["lam"], p["mu"])
    node_of, dof_of = np.full(mesh.neq, -1), np.full(mesh.neq, -1)
    j, d = np.nonzero(mesh.ID >= 0)
    node_of[mesh.ID[j, d]], dof_of[mesh.ID[j, d]] = j, d

    def at(eq):
        return torch.as_tensor(node_of[eq], device="cuda"), torch.as_tensor(dof_of[eq], device="cuda")

    sn, sd = at(p["src_eq"])
    rn, rd = at(p["eqdis"])
    ftab = torch.as_tensor(p["ftab"], device="cuda")
    zero = torch.zeros(mesh.nj, 9, S, dtype=torch.float64, device="cuda")
    x = (zero, zero, zero)
    keep = torch.as_tensor(mesh.store_nodes.astype(np.int64), device="cuda")
    hist, rec = [], []
    sh = torch.arange(S, device="cuda")
    for n in range(N + 1):
        rec.append(x[1][rn, rd])
        if case["kind"] == "evaluation":
            hist.append(x[1][keep, :3].clone())
        src = []
        for q in (0, 2, 2, 1):
            b = torch.zeros_like(zero)
            b[sn, sd, sh] = ftab[:, n, q] * E.im[sn, sd, 0]
            src.append(b)
        x = E.step(x, src, DT, False)
    rec = torch.stack(rec)                                             # [n, q, S]
    if case["kind"] != "evaluation":
        return rec.permute(2, 1, 0).contiguous()
    res = rec - torch.as_tensor(p["dis"], device="cuda").permute(2, 1, 0)
    length = np.full(S, N) if p["lengths"] is None else p["lengths"]
    if p["mask"] is not None:
        res = res * torch.as_tensor(p["mask"].astype(np.float64), device="cuda").T[None]
    steps = torch.arange(N + 1, device="cuda")[:, None, None]
    use = (steps <= torch.as_tensor(length, device="cuda")).double()
    J = float((0.5 * DT * (res ** 2 * use)[1:]).sum())
    gl = torch.zeros(mesh.nj, dtype=torch.float64, device="cuda")
    gm = torch.zeros_like(gl)
    back = torch.full((mesh.nj,), 0, dtype=torch.int64, device="cuda")
    back[keep] = torch.arange(len(keep), device="cuda")
    el = back[E.rd]
    x = (zero, zero, zero)
    for n in range(N, 0, -1):
        if n < N:
            gu = torch.stack(E._grad(el, hist[n]), dim=-2)
            gp = torch.stack(E._grad(E.rd, x[1][:, :3]), dim=-2)
            tu, tp = (g[..., 0, 0, :] + g[..., 1, 1, :] + g[..., 2, 2, :] for g in (gu, gp))
            su, sp = gu + gu.transpose(-2, -3), gp + gp.transpose(-2, -3)
            w = E.w[None, :]
            gl += E._add(E.rd, ((tu * tp).sum(-1) * w * DT).reshape(-1, 1))[:, 0]
            gm += E._add(E.rd, (0.5 * (su * sp).sum((-3, -2)).sum(-1) * w * DT).reshape(-1, 1))[:, 0]
        r1 = torch.zeros_like(zero)
        r4 = torch.zeros_like(zero)
        live = use[n]
        r1.index_put_((rn, rd), res[n] * live, accumulate=True)
        r4.index_put_((rn, rd), res[n - 1] * live, accumulate=True)
        r1, r4 = r1 * E.im, r4 * E.im
        x = E.step(x, (r1, 0.5 * (r1 + r4), 0.5 * (r1 + r4), r4), -DT, True)
    return dict(misfit=J, g_lambda=gl, g_mu=gm)


def _exact_update(case, seed):
    mesh, keep, m, g = _update_inputs(case, seed)
    E = _Exact(mesh, m[-1][0].cpu().numpy(), m[-1][1].cpu().numpy())

    def tv(v):
        gr = torch.stack([a[:, :, 0, 0] for a in E._grad(E.rd, v[:, None, None])])        # [axis, e, 27]
        num = (gr ** 2).sum(0)
        den = torch.sqrt(num + 0.01)
        reg = E._div(E.rd, [(a / den)[:, :, None, None] for a in gr])[:, 0, 0]
        return reg, float((num / den * E.w).sum())

    reg_l, cost_l = tv(m[-1][0])
    reg_m, cost_m = tv(m[-1][1])
    mass = E._add(E.rd, E.w[None, :].expand(len(E.rd), 27).reshape(-1, 1))[:, 0]
    img = torch.where(mass > 1e-10, 1.0 / torch.where(mass > 1e-10, mass, torch.ones_like(mass)), torch.zeros_like(mass))
    s_l, s_m = ((gr + 0.3 * gr.norm() / reg.norm() * reg) * img for gr, reg in ((g[-1][0], reg_l), (g[-1][1], reg_m)))
    pairs = []
    for k in range(len(m) - 1, 0, -1):                                                     # newest first
        y, s = [a - b for a, b in zip(g[k], g[k - 1])], [a - b for a, b in zip(m[k], m[k - 1])]
        ys, yy = sum((a * b).sum() for a, b in zip(y, s)), sum((a * a).sum() for a in y)
        pairs.append((y, [v * keep for v in s], 1.0 / ys, ys / yy))
    pairs = pairs[: case["memory"]]
    q, alpha = [v.clone() for v in g[-1]], []
    for y, s, rho, _ in pairs:
        alpha.append(rho * sum((a * b).sum() for a, b in zip(q, s)))
        q = [a - alpha[-1] * b for a, b in zip(q, y)]
    q = [pairs[0][3] * v for v in q]
    for (y, s, rho, _), al in zip(reversed(pairs), reversed(alpha)):
        be = rho * sum((a * b).sum() for a, b in zip(q, y))
        q = [a + (al - be) * b for a, b in zip(q, s)]
    p_l, p_m = -q[0], -q[1]
    return dict(p_l=p_l, p_m=p_m, s_l=s_l, s_m=s_m, cost_l=cost_l, cost_m=cost_m,
                slope=float((s_l * p_l).sum() + (s_m * p_m).sum()), cap_l=float(p_l.abs().max()), cap_m=float(p_m.abs().max()))


def _exact_conv(case, seed):
    x, w, b, gy = _conv_inputs(case, seed)
    ci, co, dims = case["cin"], case["cout"], (case["lz"], case["ly"], case["lx"])

    def grid(v, n):
        return v.double().cpu()[:, :n].T.reshape((1, n) + dims).contiguous()

    def rows(v, n):
        out = torch.zeros(v[0, 0].numel(), 16, dtype=torch.float64)
        out[:, :n] = v.reshape(n, -1).T
        return out

    X, W, B = grid(x, ci).requires_grad_(), w.double().cpu().reshape(co, ci, 3, 3, 3).requires_grad_(), b.double().cpu().requires_grad_()
    Y = torch.nn.functional.conv3d(X, W, B, padding=1)
    if case["kind"] == "conv_forward":
        return rows((Y.relu() if case["relu"] else Y).detach(), co)
    GY = grid(gy, co) * ((Y > 0).double() if case["relu"] else 1.0)
    gx, gw, gb = torch.autograd.grad(Y, (X, W, B), GY)
    return rows(gx, ci), gw.reshape(co, ci, 27), gb


def exact(case, seed):
    if case["kind"].startswith("conv"):
        return _exact_conv(case, seed)
    if case["kind"] == "update":
        return _exact_update(case, seed)
    passes = 2 if case["kind"] == "evaluation" else 1
    if _equations(case["nx"], case["ny"], case["nz"], case["npml"]) * case["shots"] * case["nstep"] * passes > 2.5e9:
        return None          # over about 20 seconds
    return _exact_solve(case, seed)
