"""Assembly where an entry is not where the entry before it says: distorted elements against
the oracle, and equations numbered in a random order against the lattice order, bit for bit
(the elements of an entry are added in the order of their colours either way).  Bar against
the oracle, which adds them in another order: 1e-14 of the largest entry."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from problems import RHO, tiny
from test_gpu_line import _distorted

pytestmark = pytest.mark.gpu


def _operator(mesh, p):
    from hirensi_b200.solver import Solver
    out = []
    with Solver("fp64") as s:
        s.set_mesh(mesh, RHO)
        for _ in range(2):   # with the discovery of the pattern, and with the pattern known
            s.assemble(p["lam_t"], p["mu_t"])
            out.append([s.operator_csr(w) for w in range(3)] + [s.diag_m()])
    for w in range(3):
        assert all(np.array_equal(x, y) for x, y in zip(out[0][w], out[1][w]))
    return out[1]


@pytest.mark.parametrize("size,distorted", [((4, 2, 2, 1), True), ((4, 2, 2, 2), True), ((4, 4, 2, 1), False)])
def test_assembly_matches_oracle_in_any_numbering(gpu_lib, size, distorted):
    nx, ny, nz, npml = size
    p = tiny(nx=nx, ny=ny, nz=nz, npml=npml)
    mesh = _distorted(p["mesh"]) if distorted else p["mesh"]
    got = _operator(mesh, p)
    S = O.OracleSystem.assemble(O.OracleMesh(mesh, RHO), p["lam_t"], p["mu_t"])
    perm = np.random.default_rng(2).permutation(mesh.neq)
    ID = np.where(mesh.ID >= 0, perm[np.maximum(mesh.ID, 0)], mesh.ID).astype(mesh.ID.dtype)
    moved = _operator(dataclasses.replace(mesh, ID=ID), p)
    for w in range(3):
        ia_r, ja_r, a_r = S.csr(w)
        ia, ja, a = got[w]
        assert np.array_equal(ia, ia_r) and np.array_equal(ja, ja_r), w
        assert np.max(np.abs(a - a_r)) <= 1e-14 * np.abs(a_r).max(), w
        ip, jp, b = moved[w]
        row = np.repeat(np.arange(mesh.neq), np.diff(ia))
        key = perm[row].astype(np.int64) * mesh.neq + perm[ja]
        order = np.argsort(key)
        assert np.array_equal(key[order], np.repeat(np.arange(mesh.neq), np.diff(ip)).astype(np.int64) * mesh.neq + jp)
        assert np.array_equal(a[order], b), w
    assert np.array_equal(moved[3][perm], got[3])
