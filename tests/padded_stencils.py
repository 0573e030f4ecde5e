"""Engines whose stencils are padded with members of zero weight (the cell
itself): any number of members, the sums of the stencils as they are."""
import numpy as np

from ucns3d_b200 import _native as N
from ucns3d_b200.engine import Engine


def padded_engine(m, cfg, imax, imax2=0):
    """The engine of m with imax members a stencil (CWENO: imax2 of the lower order)."""
    c = N.UcgConfig.from_buffer_copy(cfg)
    t, s = m.recon(), m.sizes
    A, n = s["admis_max"], m.ncells
    c.imax = imax
    st = np.empty((n, A, imax + 1), dtype=np.int32)
    st[:] = np.arange(n, dtype=np.int32)[:, None, None]
    st[:, :, :s["imax"] + 1] = np.where(t["stencil"] >= 0, t["stencil"], st[:, :, :s["imax"] + 1])
    M = np.zeros((t["ntables"], A, imax, s["ideg"]))
    M[:, :, :s["imax"]] = t["invmat"]
    r = N.UcgRecon.from_buffer_copy(m.recon_struct())
    r.stencil, r.invmat = N.ptr(st, N.C.c_int32), N.ptr(M, N.C.c_double)
    if s["ideg2"]:
        c.imax2 = imax2
        M2 = np.zeros((t["ntables"], A, imax2, s["ideg2"]))
        M2[:, :, :s["imax2"]] = t["invmat2"]
        r.invmat2 = N.ptr(M2, N.C.c_double)
    e = Engine(m, c, upload=False)
    e.upload_geometry(m.geometry_struct())
    e.upload_recon(r)
    return e
