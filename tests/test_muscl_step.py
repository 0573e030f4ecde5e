"""The MUSCL step: stencils of more members than k_muscl takes per pass, and
the time steps that the last stage's update forms."""
import numpy as np
import pytest

from ucns3d_b200 import _native as N
from ucns3d_b200.config import EULER, NAVIER_STOKES, make_config
from ucns3d_b200.engine import Engine
from ucns3d_b200.mesh import IC_TGV, SCHEME_MUSCL, Mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [N.UCG_FP64, N.UCG_MIXED])
@pytest.mark.parametrize("gov", [EULER, NAVIER_STOKES])
def test_muscl_more_members_than_a_pass(gov, precision):
    """MUSCL with stencils of more members than k_muscl takes per pass: the
    extra rows have zero matrices (the cell itself as member), so the result
    is that of the shorter stencil, on a cell count that leaves part of the
    last group of 32 unused."""
    m = Mesh.box_hex(7, 5, 5, periodic=(0, 1, 1), bc=(3, 3, 0, 0, 0, 0)).prepare(SCHEME_MUSCL, 1)
    if gov == NAVIER_STOKES:
        m = Mesh.box_tet(3, 3, 3, seed=9).prepare(SCHEME_MUSCL, 1)
    n, K = m.ncells, m.sizes["imax"]
    U = m.initial_condition(IC_TGV, [1.4, 5.0, 1.0])
    U = U * (1.0 + 0.02 * np.sin(2.1 * m.centres()[:, :1] + np.arange(5.0)))
    rec = m.recon()
    ref = None
    for extra in (0, 1, 11):
        cfg = make_config(m, governing=gov, precision=precision, reynolds=200.0, pres=5.0, prandtl=0.71)
        cfg.imax = K + extra
        e = Engine(m, cfg, upload=False)
        e.upload_geometry(m.geometry_struct())
        st = np.tile(np.arange(n, dtype=np.int32)[:, None], (1, K + 1 + extra))
        st[:, :K + 1] = rec["stencil"][:, 0]
        inv = np.zeros((rec["invmat"].shape[0], 1, K + extra, 3))
        inv[:, :, :K] = rec["invmat"]
        r = N.UcgRecon()
        r.first, r.count, r.ntables = 0, n, inv.shape[0]
        r.stencil, r.invmat = N.ptr(st, N.C.c_int32), N.ptr(inv, N.C.c_double)
        r.table_id = N.ptr(rec["table_id"], N.C.c_int32)
        e.upload_recon(r)
        e.set_state(U)
        R = e.residual()
        ref = R if ref is None else ref
        assert np.array_equal(R, ref), extra


@pytest.mark.parametrize("gov", [EULER, NAVIER_STOKES])
def test_time_steps_formed_by_the_last_stage(gov):
    """ucg_step forms each following step's CFL time step in the last stage's
    update: the same steps as CALCULATE_CFL and RK3 called one by one, also
    when calls follow one another and other calls use the time step between."""
    m = Mesh.box_tet(4, 4, 3, seed=2).prepare(SCHEME_MUSCL, 1)
    cfg = make_config(m, governing=gov, reynolds=200.0, pres=5.0, prandtl=0.71)
    U = m.initial_condition(IC_TGV, [1.4, 5.0, 1.0])
    a, b = Engine(m, cfg), Engine(m, cfg)
    a.set_state(U)
    b.set_state(U)
    for nsteps, cfl in ((1, 0.5), (2, 0.4), (5, 0.3), (0, 0.3), (3, 0.5)):
        a.time_marching(nsteps, cfl)
        for _ in range(nsteps):
            dt = b.calculate_cfl(cfl)
            b.runge_kutta3(dt)
        assert a.last_dt() == dt
        assert np.array_equal(a.get_state(), b.get_state())
        assert a.calculate_cfl(0.2) == b.calculate_cfl(0.2) == a.last_dt()
        dt = a.last_dt()
