"""Matrix sets shared by many cells (k_lsq_set, k_wis_set, k_adj_lsq_set):
the same engine once with the tables of one upload, whose shared sets are
tiled, and once with the same tables uploaded in two halves, where every cell
reads its own copy.  The forward kernels take the same operations in the same
order, so residuals and states are equal bit for bit; the reverse adds a
member's rows and a cell's stencils in another order (FP64 rounding of sums of
at most a few thousand terms of one size: 1e-12 of the result's largest value).

Meshes: whole tiles and remainders (1 to 127 cells in a set's last tile), sets
above and below the 32 cells from which they are tiled, all cells tiled and
some left over (a box without periodicity), CWENO with both stencil sizes,
renumbered cells, Navier-Stokes."""
import numpy as np
import pytest

from ucns3d_b200 import _native as N
from ucns3d_b200.config import EULER, NAVIER_STOKES, make_config
from ucns3d_b200.engine import Engine, EngineError
from ucns3d_b200.mesh import IC_TGV, SCHEME_MUSCL, SCHEME_WENO, Mesh, RenumberedMesh

pytestmark = pytest.mark.gpu

CASES = {
    "weno5_hex12": (lambda: Mesh.box_hex(12, 12, 12), SCHEME_WENO, 4, 0, EULER, 1),
    "weno5_hex_open": (lambda: Mesh.box_hex(10, 10, 24, periodic=(1, 1, 0), bc=(0, 0, 0, 0, 6, 6)), SCHEME_WENO, 4, 0,
                       EULER, 1),
    "weno5_hex_char": (lambda: Mesh.box_hex(11, 10, 10), SCHEME_WENO, 4, 0, EULER, 2),
    "weno3_ns_hex9": (lambda: Mesh.box_hex(9, 9, 9), SCHEME_WENO, 2, 0, NAVIER_STOKES, 1),
    "weno3_tet": (lambda: Mesh.box_tet(10, 10, 10, jitter=0.0), SCHEME_WENO, 2, 0, EULER, 1),
    "cweno4_ns_mixed10": (lambda: Mesh.mixed_box(10, seed=4), SCHEME_WENO, 3, 5, NAVIER_STOKES, 1),
    "cweno4_mixed16": (lambda: Mesh.mixed_box(16, seed=1234), SCHEME_WENO, 3, 5, EULER, 1),
    "cweno4_ns_mixed16": (lambda: Mesh.mixed_box(16, seed=1234), SCHEME_WENO, 3, 5, NAVIER_STOKES, 1),
    "cweno4_char_mixed10": (lambda: Mesh.mixed_box(10, seed=4), SCHEME_WENO, 3, 5, EULER, 2),
    "muscl_p2_hex8": (lambda: Mesh.box_hex(8, 8, 8), SCHEME_MUSCL, 2, 0, EULER, 1),
}
PARTLY = ("weno5_hex_open", "cweno4_mixed16", "cweno4_ns_mixed16")  # some cells are left over


def _engines(name, precision, shuffle=False):
    mk, scheme, iorder, ees, gov, wenwrt = CASES[name]
    m = mk().prepare(scheme, iorder, ees)
    if shuffle:
        m = RenumberedMesh(m, np.random.default_rng(5).permutation(m.ncells))
    cfg = make_config(m, governing=gov, precision=precision, reynolds=200.0, pres=5.0, prandtl=0.71, wenwrt=wenwrt)
    shared = Engine(m, cfg)
    own = Engine(m, cfg, upload=False)
    own.upload_geometry(m.geometry_struct())
    r, s, n = m.recon_struct(), m.sizes, m.ncells
    row = s["admis_max"] * (s["imax"] + 1)
    st = np.ctypeslib.as_array(r.stencil, shape=(n * row,))
    tid = np.ctypeslib.as_array(r.table_id, shape=(n,))
    half = n // 2
    for a, b in ((0, half), (half, n)):
        part = N.UcgRecon.from_buffer_copy(r)
        part.first, part.count = a, b - a
        part.stencil = N.ptr(st[a * row:b * row], N.C.c_int32)
        part.table_id = N.ptr(tid[a:b], N.C.c_int32)
        own.upload_recon(part)
    x = m.centres()
    U = m.initial_condition(IC_TGV, [1.4, 5.0, 1.0])
    U = U * (1.0 + 0.02 * np.sin(1.3 * x[:, :1] + 0.7 * x[:, 1:2] + 2.1 * x[:, 2:3] + np.arange(5.0)))
    return m, shared, own, U


@pytest.mark.parametrize("precision", [N.UCG_FP64, N.UCG_MIXED])
@pytest.mark.parametrize("name", list(CASES))
def test_shared_sets_equal_own_tables(name, precision):
    m, shared, own, U = _engines(name, precision, shuffle=name in ("weno5_hex12", "cweno4_ns_mixed10"))
    cells = shared.shared_sets()["cells"]
    assert own.shared_sets() == {"cells": 0, "sets": 0}
    assert cells == m.ncells if name not in PARTLY else 0 < cells < m.ncells
    out = []
    for e in (shared, own):
        e.set_state(U)
        R = e.residual()
        e.time_marching(2, 0.4)
        out.append((R, e.get_state(), e.last_dt()))
        e.check_health()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]
    assert np.abs(out[0][0]).max() > 0


@pytest.mark.parametrize("name", ["weno5_hex12", "weno5_hex_open", "weno3_ns_hex9", "weno3_tet", "cweno4_ns_mixed10",
                                  "cweno4_mixed16"])
def test_shared_sets_reverse(name):
    m, shared, own, U = _engines(name, N.UCG_FP64, shuffle=name == "weno3_tet")
    rng = np.random.default_rng(3)
    lam, du = rng.standard_normal(U.shape), rng.standard_normal(U.shape) * 1e-2
    out = []
    for e in (shared, own):
        e.set_state(U)
        mu, pbar = e.residual_vjp(lam)
        out.append((mu, pbar, e.residual_jvp(du)))
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-12 * max(np.abs(b).max(), 1e-300)
    assert np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("precision", [N.UCG_FP64, N.UCG_MIXED])
@pytest.mark.parametrize("name", ["weno5_hex12", "weno5_hex_open", "cweno4_ns_mixed10"])
def test_wait_timeout_is_reported_and_recoverable(name, precision, monkeypatch):
    """The bounded waits between the warps of k_lsq_set (and of k_lsq_ring for
    the cells left over): with a limit of 0 polls every wait gives up and the
    kernels return, ucg_check_health reports UCG_ETIMEOUT, and with the default
    limit restored the handle gives its residual again, bit for bit."""
    monkeypatch.setenv("UCG_LSQ_WAIT", "1")
    m, e, own, U = _engines(name, precision)
    own.close()
    e.set_state(U)
    ref = e.residual()
    e.check_health()
    assert e.lib.ucg_set_wait_limit(e._h, 0) == N.UCG_OK
    e.residual()
    with pytest.raises(EngineError) as ei:
        e.check_health()
    assert ei.value.code == N.UCG_ETIMEOUT
    assert e.lib.ucg_set_wait_limit(e._h, -1) == N.UCG_OK
    assert np.array_equal(e.residual(), ref)
    e.check_health()


@pytest.mark.parametrize("precision", [N.UCG_FP64, N.UCG_MIXED])
@pytest.mark.parametrize("ees", [0, 5])
@pytest.mark.parametrize("mesh", ["hex", "hex_large", "tet", "mixed"])
def test_iorder1_large_meshes(mesh, ees, precision, monkeypatch):
    """IORDER 1 from 128 cells per SM on: the least squares one lane per cell
    (k_lsq_lane) against the ring (UCG_LSQ_BULK=1), bit for bit.  Tiles only
    without CWENO, below 512 cells per SM and where the cells of a set follow
    one another (a box of hexahedra)."""
    import torch

    mk = {"hex": lambda: Mesh.box_hex(27, 27, 29), "tet": lambda: Mesh.box_tet(15, 15, 15, seed=2),
          "hex_large": lambda: Mesh.box_hex(43, 43, 41), "mixed": lambda: Mesh.mixed_box(20, seed=4)}[mesh]
    m = mk().prepare(SCHEME_WENO, 1, ees)
    per_sm = m.ncells / torch.cuda.get_device_properties(0).multi_processor_count
    assert per_sm >= 512 if mesh == "hex_large" else 128 <= per_sm < 512
    cfg = make_config(m, governing=EULER, precision=precision, pres=5.0)
    x = m.centres()
    U = m.initial_condition(IC_TGV, [1.4, 5.0, 1.0])
    U = U * (1.0 + 0.02 * np.sin(1.3 * x[:, :1] + 0.7 * x[:, 1:2] + 2.1 * x[:, 2:3] + np.arange(5.0)))
    out = []
    for bulk in ("0", "1"):
        monkeypatch.setenv("UCG_LSQ_BULK", bulk)
        e = Engine(m, cfg)
        assert e.shared_sets()["cells"] == (m.ncells if mesh == "hex" and not ees and bulk == "0" else 0)
        e.set_state(U)
        r = [e.residual()]
        if precision == N.UCG_FP64:
            r.append(e.residual_jvp(U * 1e-2))
        e.check_health()
        e.close()
        out.append(r)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
