"""The MUSCL adjoint's forward records (k_adj_fwd) and tangent (k_jvp_muscl),
one warp per variable of a 32-cell group: cell counts that leave 29, 1 or no
cells of the last group unused, stencils of eight members (one pass of the
viscous records) and of more, walls.  The reverse is the transpose of the tangent (sums of a few
thousand terms in FP64: 1e-12 of the terms' size), and the tangent is the
derivative of the residual (central differences with step 1e-6: rounding
1e-10 and truncation 1e-12 of the residual's derivative; the median, since a
cell whose limiter switches within the step has no derivative)."""
import numpy as np
import pytest

from ucns3d_b200 import _native as N
from ucns3d_b200.config import EULER, NAVIER_STOKES, make_config
from ucns3d_b200.engine import Engine
from ucns3d_b200.mesh import IC_TGV, SCHEME_MUSCL, Mesh

pytestmark = pytest.mark.gpu

MESHES = {
    "hex_99": lambda: Mesh.box_hex(11, 3, 3, periodic=(0, 1, 1), bc=(4, 4, 0, 0, 0, 0)),
    "hex_63": lambda: Mesh.box_hex(7, 3, 3),
    "hex_64": lambda: Mesh.box_hex(4, 4, 4),
    "tet_162": lambda: Mesh.box_tet(3, 3, 3, seed=9),
    "mixed_540": lambda: Mesh.mixed_box(6, seed=4),
}


def _setup(name, gov):
    m = MESHES[name]().prepare(SCHEME_MUSCL, 1)
    cfg = make_config(m, governing=gov, reynolds=50.0, pres=5.0, prandtl=0.71)
    x = m.centres()
    U = m.initial_condition(IC_TGV, [1.4, 5.0, 1.0])
    U = U * (1.0 + 0.02 * np.sin(1.3 * x[:, :1] + 0.7 * x[:, 1:2] + 2.1 * x[:, 2:3] + np.arange(5.0)))
    rng = np.random.default_rng(8)
    return m, cfg, U, rng.standard_normal(U.shape), rng.standard_normal(U.shape) * 1e-2


@pytest.mark.parametrize("gov", [EULER, NAVIER_STOKES])
@pytest.mark.parametrize("name", list(MESHES))
def test_reverse_and_tangent(name, gov):
    m, cfg, U, lam, du = _setup(name, gov)
    e = Engine(m, cfg)
    e.set_state(U)
    mu = e.residual_vjp(lam)[0]
    tang = e.residual_jvp(du)
    assert abs((mu * du).sum() - (lam * tang).sum()) <= 1e-12 * (np.abs(mu * du).sum() + np.abs(lam * tang).sum())
    h = 1e-6
    R = []
    for s in (h, -h):
        e.set_state(U + s * du)
        R.append(e.residual())
    fd = (R[0] - R[1]) / (2 * h)
    assert np.median(np.abs(tang - fd)) <= 1e-7 * np.abs(fd).max()
    e.check_health()


@pytest.mark.parametrize("gov", [EULER, NAVIER_STOKES])
def test_more_members_than_a_pass(gov):
    """Extra stencil rows of zero matrices (the cell itself as member) change
    nothing, whichever pass they fall into."""
    m, cfg, U, lam, du = _setup("tet_162", gov)
    n, K, rec, ref = m.ncells, m.sizes["imax"], m.recon(), None
    for extra in (0, 1, 11):
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
        out = (*e.residual_vjp(lam), e.residual_jvp(du))
        ref = out if ref is None else ref
        for a, b in zip(out, ref):
            assert np.array_equal(a, b), extra
