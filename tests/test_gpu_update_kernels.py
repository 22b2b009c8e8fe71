"""Kernels of the model update at the edges of their blocks: reductions around one block and
the full grid, TV on element counts that leave a block part empty, and the L-BFGS chain with
memories of one, two and several pairs on vectors shorter and longer than its grid.  Bars:
FP64 sums of n terms in any order agree within n 2^-53 of the sum of magnitudes; the
direction is a few such sums deep, relative L2 1e-11."""
import numpy as np
import pytest

import oracle as O
from hirensi_b200.inversion import DeviceBackend
from hirensi_b200.mesh import box_mesh
from problems import RHO, rel_l2

pytestmark = pytest.mark.gpu


def _backend(nx, ny, nz, npml):
    from hirensi_b200.solver import Solver
    mesh = box_mesh(nx, ny, nz, 1.25, npml)
    s = Solver("fp64")
    s.set_mesh(mesh, RHO)
    return s, mesh, DeviceBackend(s, mesh)


def test_reductions_at_block_edges(gpu_lib):
    s, _, dev = _backend(2, 2, 2, 1)
    rng = np.random.default_rng(3)
    for n in (1, 2, 31, 32, 255, 256, 257, 296 * 256 - 1, 296 * 256, 296 * 256 + 1, 300001):
        x, y = rng.standard_normal(n), rng.standard_normal(n)
        X, Y = dev.vec(x), dev.vec(y)
        dev.n = n
        eps = (n + 2) * 2.0 ** -53
        assert abs(dev.dot(X, Y) - x @ y) <= 2 * eps * (np.abs(x) @ np.abs(y))
        assert abs(dev.norm2(X) - np.linalg.norm(x)) <= 2 * eps * np.linalg.norm(x)
        assert dev.norminf(X) == np.abs(x).max()
    dev.n = 0
    assert dev.dot(X, Y) == 0.0 and dev.norm2(X) == 0.0 and dev.norminf(X) == 0.0
    dev.n = 3
    assert np.isnan(dev.dot(dev.vec([1.0, np.nan, 2.0]), dev.vec([1.0, 1.0, 1.0])))
    assert dev.norminf(dev.vec([1.0, -np.inf, 2.0])) == np.inf
    s.close()


@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (3, 3, 1), (2, 2, 2), (5, 3, 3)])
def test_tv_matches_oracle(gpu_lib, nx, ny, nz):
    s, mesh, dev = _backend(nx, ny, nz, 1)
    rng = np.random.default_rng(nx)
    lam, mu = 80.0 + rng.standard_normal(mesh.nj), 40.0 + rng.standard_normal(mesh.nj)
    om = O.OracleMesh(mesh, RHO)
    rl, rm, cl, cm = O.tv_reg(om, lam, mu)
    RL, RM = dev.zeros(), dev.zeros()
    for _ in range(2):   # the finished-block count returns to zero
        dcl, dcm = dev.tv(dev.vec(lam), dev.vec(mu), RL, RM)
        assert rel_l2(dev.host(RL), rl) < 1e-12 and rel_l2(dev.host(RM), rm) < 1e-12
        assert abs(dcl - cl) < 1e-12 * abs(cl) and abs(dcm - cm) < 1e-12 * abs(cm)
    s.close()


@pytest.mark.parametrize("size,memory", [((2, 2, 2, 1), 1), ((2, 2, 2, 1), 2), ((3, 2, 2, 1), 7), ((24, 24, 12, 6), 3)])
def test_lbfgs_chain_matches_oracle(gpu_lib, size, memory):
    s, mesh, dev = _backend(*size)
    n = mesh.nj
    rng = np.random.default_rng(memory)
    keep = (rng.random(n) < 0.7).astype(np.float64)
    dev.lbfgs_setup(memory, dev.vec(keep))
    ref = O.LBFGSCoupled(n, memory, keep)
    A = 1.0 + rng.random((2, n))   # gradients of a convex quadratic: y.s > 0
    m_pre = [np.zeros(n), np.zeros(n)]
    g_pre = [np.zeros(n), np.zeros(n)]
    for it in range(1, 2 * memory + 3):
        m = [v + rng.standard_normal(n) for v in m_pre]
        g = [A[k] * m[k] for k in range(2)]
        pl, pm = ref.direction(it, 1, *g, *g_pre, *m, *m_pre)
        P = [dev.zeros(), dev.zeros()]
        dev.lbfgs_direction(it, 1, *[dev.vec(v) for v in (*g, *g_pre, *m, *m_pre)], *P)
        assert rel_l2(dev.host(P[0]), pl) < 1e-11 and rel_l2(dev.host(P[1]), pm) < 1e-11, it
        g_pre, m_pre = g, m
    s.close()
