"""Face values one warp per conserved variable below IORDER 4 (k_wface, then
k_wpost's MUSCL fall-back of the cells it flags) against one lane per cell
(k_wpost, UCG_WENO_FACE=0), bit for bit: both take the same operations in the
same order.  Cell counts leave part of the last group of 32 unused; the cells
beside a pressure jump take the fall-back; meshes on both sides of the rule
(wface_own), beyond which both engines run k_wpost: more than 128 cells per SM
at IORDER 3, 192 at IORDER 1 (FP64; never in the mixed form) and 2 (mixed form)."""
import numpy as np
import pytest

from ucns3d_b200 import _native as N
from ucns3d_b200.config import EULER, NAVIER_STOKES, make_config
from ucns3d_b200.engine import Engine
from ucns3d_b200.mesh import IC_TGV, SCHEME_WENO, Mesh

pytestmark = pytest.mark.gpu

CASES = {
    "weno3_tet": (lambda: Mesh.box_tet(5, 5, 5, seed=3), 2, 0, EULER, {}),
    "weno3_ns_hex": (lambda: Mesh.box_hex(7, 5, 5, periodic=(0, 1, 1), bc=(3, 3, 0, 0, 0, 0)), 2, 0, NAVIER_STOKES, {}),
    "cweno3_mixed": (lambda: Mesh.mixed_box(6, seed=4), 2, 5, EULER, {}),
    "cweno4_ns_mixed": (lambda: Mesh.mixed_box(10, seed=4), 3, 5, NAVIER_STOKES, {}),
    "cweno4_z_tet": (lambda: Mesh.box_tet(7, 7, 7, seed=9), 3, 5, EULER, {"wenoz": 1}),
    "weno4_hex": (lambda: Mesh.box_hex(9, 9, 11), 3, 0, EULER, {}),
    "weno4_hex_large": (lambda: Mesh.box_hex(28, 28, 25), 3, 0, EULER, {}),
    "weno2_tet": (lambda: Mesh.box_tet(5, 5, 5, seed=3), 1, 0, EULER, {}),
    "cweno2_hex": (lambda: Mesh.box_hex(9, 9, 11), 1, 5, EULER, {}),
    "weno2_hex_large": (lambda: Mesh.box_hex(31, 31, 31), 1, 0, EULER, {}),
    "weno3_hex_large": (lambda: Mesh.box_hex(31, 31, 31), 2, 0, EULER, {}),
}


def _lanes(name, precision):
    """Both engines take one lane per cell."""
    return (name in ("weno4_hex_large", "weno2_hex_large") or
            (precision == N.UCG_MIXED and name in ("weno2_tet", "cweno2_hex", "weno3_hex_large")))


@pytest.mark.parametrize("precision", [N.UCG_FP64, N.UCG_MIXED])
@pytest.mark.parametrize("jump", [False, True])
@pytest.mark.parametrize("name", list(CASES))
def test_warp_per_variable_equals_lane_per_cell(name, jump, precision, monkeypatch):
    mk, iorder, ees, gov, more = CASES[name]
    m = mk().prepare(SCHEME_WENO, iorder, ees)
    cfg = make_config(m, governing=gov, precision=precision, reynolds=200.0, pres=5.0, prandtl=0.71, **more)
    x = m.centres()
    U = m.initial_condition(IC_TGV, [1.4, 5.0, 1.0])
    if jump:
        left = x[:, 0] < 0.5 * (x[:, 0].min() + x[:, 0].max())
        U[:] = 0.0
        U[:, 0], U[:, 4] = np.where(left, 1.0, 0.125), np.where(left, 1.0, 0.05) / 0.4
    else:
        U = U * (1.0 + 0.02 * np.sin(1.3 * x[:, :1] + 0.7 * x[:, 1:2] + 2.1 * x[:, 2:3] + np.arange(5.0)))
    out, launches = [], []
    for flag in ("1", "0"):
        monkeypatch.setenv("UCG_WENO_FACE", flag)
        e = Engine(m, cfg)
        e.set_state(U)
        before = e.launch_count
        out.append(e.residual())
        launches.append(e.launch_count - before)
        e.check_health()
        e.close()
    assert np.array_equal(out[0], out[1])
    # the fall-back is a launch of its own behind k_wface
    assert launches[0] - launches[1] == (0 if _lanes(name, precision) else 1)
