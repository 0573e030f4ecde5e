"""Stencils of any number of members: the matrix sets that many cells share are
kept in shared memory only where their rows fit (plan_sets); with more members
every cell reads its own tables.  A stencil padded with members of zero weight
gives the sums of the stencil itself, so the residual, the states and the
derivatives equal those of the unpadded engine bit for bit (reverse: up to the
order of its sums, 1e-12), on both sides of each limit."""
import numpy as np
import pytest

from padded_stencils import padded_engine
from ucns3d_b200 import _native as N
from ucns3d_b200.config import EULER, NAVIER_STOKES, make_config
from ucns3d_b200.engine import Engine
from ucns3d_b200.mesh import IC_TGV, SCHEME_WENO, Mesh

pytestmark = pytest.mark.gpu

# members at which the rows of 34 (19) values and the 5,120 gathered differences
# of k_lsq_set's rings still fit in 226 KB, in 8 or 4 bytes
FIT = {(4, N.UCG_FP64): (226 * 1024 - 5120 * 8) // (34 * 8), (4, N.UCG_MIXED): (226 * 1024 - 5120 * 4) // (36 * 4),
       (3, N.UCG_FP64): (226 * 1024 - 5120 * 8) // (20 * 8)}


@pytest.mark.parametrize("iorder,ees,gov,precision,over", [
    (4, 0, EULER, N.UCG_FP64, 0), (4, 0, EULER, N.UCG_FP64, 1), (4, 0, EULER, N.UCG_FP64, 40),
    (4, 0, EULER, N.UCG_MIXED, 0), (4, 0, EULER, N.UCG_MIXED, 1), (4, 0, EULER, N.UCG_MIXED, 80),
    (3, 5, NAVIER_STOKES, N.UCG_FP64, 0), (3, 5, NAVIER_STOKES, N.UCG_FP64, 1),
    (3, 5, NAVIER_STOKES, N.UCG_FP64, 60)])
def test_padded_stencils(iorder, ees, gov, precision, over):
    m = Mesh.box_hex(5, 5, 5).prepare(SCHEME_WENO, iorder, ees)
    cfg = make_config(m, governing=gov, precision=precision, reynolds=200.0, pres=5.0, prandtl=0.71)
    imax = FIT[iorder, precision] + over
    x = m.centres()
    U = m.initial_condition(IC_TGV, [1.4, 5.0, 1.0])
    U = U * (1.0 + 0.02 * np.sin(1.3 * x[:, :1] + 0.7 * x[:, 1:2] + np.arange(5.0)))
    lam = np.random.default_rng(3).standard_normal(U.shape)
    out = []
    for e in (Engine(m, cfg), padded_engine(m, cfg, imax, imax)):
        e.set_state(U)
        r = [e.residual()]
        e.time_marching(1, 0.4)
        r.append(e.get_state())
        if precision == N.UCG_FP64:
            e.set_state(U)
            r += [e.residual_jvp(lam), e.residual_vjp(lam)[0]]
        e.check_health()
        e.close()
        out.append(r)
    for k, (a, b) in enumerate(zip(*out)):
        assert np.abs(b).max() > 0
        if k < 3:
            assert np.array_equal(a, b)
        else:
            assert np.abs(a - b).max() <= 1e-12 * np.abs(a).max()
