"""The line operator with uneven records and checkpoints, and the kernel that keeps an element
in one thread's registers where every element is loaded.

Bars.  FP64 variants of the same steps: 1e-11 (their sums differ in order only).  FP32
against FP64 over 12 steps: 48 stages of about ten roundings each, independent of one
another, leave sqrt(480) 2^-24 = 1.3e-6 of the fields and twice that of their products;
1e-5 here.  A load on every fifth node puts a value of the same order into every element, so
that one wrong element of 7560 changes the fields by 1e-2."""
import numpy as np
import pytest

from problems import RHO, rel_l2, tiny
from test_gpu_uneven import LENS, _batch, _data, _masks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,ckpt", [(96, 0), (97, 17), (98, 9)])
def test_uneven_records(gpu_lib, variant, ckpt):
    p = tiny(nshot=3, nstep=max(LENS))
    dis, mask = _data(p), _masks(p)
    J0, gl0, gm0, tr0 = _batch(p, dis, mask, variant=41)
    J1, gl1, gm1, tr1 = _batch(p, dis, mask, variant=variant, ckpt=ckpt)
    assert abs(J1 - J0) <= 1e-11 * J0
    assert rel_l2(gl1, gl0) < 1e-11 and rel_l2(gm1, gm0) < 1e-11 and rel_l2(tr1, tr0) < 1e-11


@pytest.mark.parametrize("nshot,variant,ckpt", [(8, 98, 0), (7, 96, 5), (8, 97, 4)])
def test_register_elements_with_every_element_loaded(gpu_lib, nshot, variant, ckpt):
    from hirensi_b200.configs import inversion_config
    from hirensi_b200.solver import Solver
    p = inversion_config(nstep=12, nx=21, ny=20, nz=18, npml=1, shots=tuple((2.5 * k - 10.0, 5.0) for k in range(nshot)),
                         receivers=(-10.0, 0.0, 10.0), fr=900.0)
    rng = np.random.default_rng(2)
    src = p.mesh.equations(p.mesh.store_nodes[::5])
    b = rng.standard_normal((src.size, nshot))
    dis = 1e-6 * rng.standard_normal((nshot, len(p.eqdis), p.nstep + 1))
    out = {}
    for prec, v in (("fp32", variant), ("fp64", 41)):
        with Solver(prec) as s:
            s.set_mesh(p.mesh, RHO)
            s.assemble(p.lam_true, p.mu_true)
            s.set_history(p.mesh.store_eq)
            s.set_shots(p.nstep, p.dt, src, b, p.ftab)
            s.set_receivers(p.eqdis, p.eqdis_map)
            s.set_variant(v, v)
            s.set_checkpointing(ckpt)
            s.forward()
            s.misfit(dis)
            fields = [s.state(2 * ckpt, k)[1] if ckpt else s.history(k)[-1] for k in (0, nshot - 1)]
            out[prec] = fields + [s.traces(), *s.adjoint_gradient(dis)]
    for a, c in zip(out["fp32"], out["fp64"]):
        assert np.abs(c).max() > 0 and rel_l2(a, c) < 1e-5
