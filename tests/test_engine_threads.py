"""Engines on two host threads (one thread per handle).  A kernel's limit of
dynamic shared memory belongs to the device's context and not to an engine, so
two engines that ask different amounts of the same kernel must not be able to
refuse each other's launches: stencils of different length, with and without
shared matrix sets (the reverse kernels hold a set's triangles), tables built on
the device at different orders.  The threads repeat their calls until the
launches have met many times; every result equals the first one, bit for bit."""
import threading

import numpy as np
import pytest

from padded_stencils import padded_engine
from ucns3d_b200.config import EULER, make_config
from ucns3d_b200.engine import Engine
from ucns3d_b200.mesh import IC_TGV, SCHEME_WENO, Mesh

pytestmark = pytest.mark.gpu


def _together(*calls):
    """Each (call, repeats) on a thread of its own; what went wrong in any."""
    errors = []
    start = threading.Barrier(len(calls))

    def work(call, repeats):
        try:
            ref = call()
            start.wait()
            for _ in range(repeats):
                if errors:
                    return
                for a, b in zip(ref, call()):
                    assert np.array_equal(a, b)
        except Exception as err:  # noqa: BLE001 - reported by the test
            errors.append(err)
            start.abort()

    threads = [threading.Thread(target=work, args=c) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def _hex(n=5):
    m = Mesh.box_hex(n, n, n).prepare(SCHEME_WENO, 4, 0)
    x = m.centres()
    U = m.initial_condition(IC_TGV, [1.4, 5.0, 1.0])
    return m, make_config(m, governing=EULER, pres=5.0), U * (1.0 + 0.02 * np.sin(1.3 * x[:, :1] + np.arange(5.0)))


def test_stencils_of_different_length():
    m, cfg, U = _hex()
    es = [Engine(m, cfg), padded_engine(m, cfg, 400)]

    def march(e):
        e.set_state(U)
        e.time_marching(40, 0.4)
        return (e.get_state(),)

    _together(*(((lambda e=e: march(e)), 60) for e in es))
    for e in es:
        e.check_health()


def test_reverse_with_and_without_shared_sets(monkeypatch):
    m, cfg, U = _hex()
    es = []
    for own in ("0", "1"):
        monkeypatch.setenv("UCG_LSQ_BULK", own)
        es.append(Engine(m, cfg))
        es[-1].set_state(U)
    lam = np.random.default_rng(1).standard_normal(U.shape)
    _together(*(((lambda e=e: (e.residual_vjp(lam)[0], e.residual_jvp(lam))), 500) for e in es))
    for e in es:
        e.check_health()


def test_device_tables_at_two_orders():
    def build(n, iorder):
        m = Mesh.box_hex(n, n, n).prepare(SCHEME_WENO, iorder, 0, tables=False)
        cfg = make_config(m, governing=EULER, pres=5.0)
        U = m.initial_condition(IC_TGV, [1.4, 5.0, 1.0])

        def call():
            e = Engine(m, cfg, tables="device")
            e.set_state(U)
            r = e.residual()
            e.close()
            return (r,)

        return call

    _together((build(6, 4), 80), (build(4, 1), 160))
