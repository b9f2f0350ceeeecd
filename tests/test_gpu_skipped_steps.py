"""Steps that are issued but do not run: the engine issues steps ahead of the
device, so those behind a stop (tstop, tmax) or behind a step whose dt choice
the host has to complete do nothing when they reach the device.  User hooks
are called for them all the same, and must leave the state alone: runs with
hooks against the FP64 oracle, bit for bit, through stops and through gas
without pressure whose flow along x alone gives no wave speed along y (every
step's dt then needs the cell-centred pass)."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from tests import test_special_bound as tb
from tests import test_special_source as ts
from vac_gb300 import inistate
from vac_gb300.engine import Engine

pytestmark = pytest.mark.gpu


def same(a, b):
    return np.array_equal(a.view(np.uint64), b.view(np.uint64))


def dust(nx=24, ny=17):
    """Gas of gamma = 1, whose pressure (gamma-1)*(...) is zero, flowing along
    x: a wave speed along x and none along y."""
    x = inistate.domain_grid((nx, ny), (0.0, 0.0), (1.0, 1.0))
    rho = 1.0 + 0.2 * np.sin(2 * np.pi * x[0]) * np.cos(2 * np.pi * x[1])
    m1 = rho * (0.3 + 0.1 * np.cos(2 * np.pi * x[0]))
    w = np.stack([rho, m1, np.zeros_like(rho), np.ones_like(rho)])
    return inistate._snap(x, w, 1.0, False, 2, "dust")


STOP_CASES = [
    ("sod", lambda: inistate.sod_1d(64), "cont"),
    ("ot", lambda: inistate.orszag_tang(24), "periodic"),
    ("rm3", lambda: inistate.random_modes(10, seed=2, p0=0.5), "periodic"),
]


@pytest.mark.parametrize("dt_hook", [False, True])
@pytest.mark.parametrize("name,mk,bc", STOP_CASES, ids=[c[0] for c in STOP_CASES])
def test_source_hook_leaves_the_state_at_a_stop(gpu_lib, name, mk, bc, dt_hook):
    Lh, hs, hd = ts._host_hook()
    Ld, ds, dd = ts._device_hook()
    s = mk()
    p = inistate.params_for(s, limiter="woodward", bc=bc)
    src = (ds, dd if dt_hook else None, None)
    e = Engine(p, s.x, s.w, source=src)
    e.step(5)
    tstop = 0.999 * e.t
    e = Engine(p, s.x, s.w, source=src)
    o = Oracle(p, s.x, s.w, source=(hs, hd if dt_hook else None, ts._e_index(p)))
    assert not e.step(13, tstop=tstop) and e.it == 5
    o.step(5)
    assert e.t == o.t and same(e.state(), o.state())
    e.step(4)
    o.step(4)
    assert (e.it, e.t) == (9, o.t) and same(e.state(), o.state())
    # the run's end likewise
    p.tmax = tstop
    e = Engine(p, s.x, s.w, source=src)
    o = Oracle(p, s.x, s.w, source=(hs, hd if dt_hook else None, ts._e_index(p)))
    assert e.step(12) and e.it == 5
    o.step(12)
    assert e.t == o.t and same(e.state(), o.state())


def test_source_hook_where_every_step_needs_the_passes(gpu_lib):
    Lh, hs, hd = ts._host_hook()
    Ld, ds, dd = ts._device_hook()
    s = dust()
    p = inistate.params_for(s)
    e = Engine(p, s.x, s.w, source=(ds, None, None))
    o = Oracle(p, s.x, s.w, source=(hs, None, ts._e_index(p)))
    e.step(12)
    o.step(12)
    assert (e.it, e.t) == (12, o.t) and same(e.state(), o.state())


def test_special_faces_keep_their_time_at_a_stop(gpu_lib):
    """The ghost values of a time-dependent 'special' face after a stop are
    those of the stop's time, also where steps issued behind it filled the
    face again."""
    Lh, hfn = tb._host_hook()
    Ld, dfn = tb._device_hook()
    s = inistate.riemann_2d(32, 3)
    p = inistate.params_for(s, bc="cont")
    tb._special([0])(p)
    # (a step after an even it starts with the x sweep, which reads the face)
    e = Engine(p, s.x, s.w, bound=(dfn, None))
    e.step(6)
    tstop = 0.999 * e.t
    e = Engine(p, s.x, s.w, bound=(dfn, None))
    o = Oracle(p, s.x, s.w, bound=(hfn, None))
    assert not e.step(13, tstop=tstop) and e.it == 6
    e.step(4)
    o.step(10)
    assert (e.it, e.t) == (10, o.t) and same(e.state(), o.state())


def test_special_faces_where_every_step_needs_the_passes(gpu_lib):
    Lh, hfn = tb._host_hook()
    Ld, dfn = tb._device_hook()
    s = dust()
    p = inistate.params_for(s, bc="cont")
    tb._special([0], ivars=[0])(p)
    e = Engine(p, s.x, s.w, bound=(dfn, None))
    o = Oracle(p, s.x, s.w, bound=(hfn, None))
    e.step(12)
    o.step(12)
    assert (e.it, e.t) == (12, o.t) and same(e.state(), o.state())


def test_removed_dt_hook_limits_nothing(gpu_lib):
    """Without the getdt_special hook its last limit no longer counts."""
    from vac_gb300.engine import _ck, lib
    Lh, hs, hd = ts._host_hook()
    Ld, ds, dd = ts._device_hook()
    s = inistate.orszag_tang(24)
    p = inistate.params_for(s)
    e = Engine(p, s.x, s.w, source=(None, dd, None))
    e.step(3)
    w = e.state()
    _ck(lib().vacgpu_register_source_fn(e.h, None, None, None), "vacgpu_register_source_fn")
    e.step(1)
    limited = 0.05 / (0.001 + np.abs(w[1] / w[0]).max())
    assert e.dt > 1.2 * limited
