"""The device-resident time loop: the dt choice at the end of the step before
against the oracle's loop -- calls of any length, stops inside a call, and
steps that need the cell-centred passes again because no wave speed set a
dt -- on FP64 grids bit for bit, and on mixed ones between call lengths."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from vac_gb300 import abi, inistate
from vac_gb300.engine import Engine, Server

pytestmark = pytest.mark.gpu


def same(a, b):
    return np.array_equal(a.view(np.uint64), b.view(np.uint64))


def gas_at_rest():
    """Uniform gas without pressure: every wave speed is zero, so each step's
    dt comes from the cell-centred passes (dt = 1e99)."""
    s = inistate.sod_1d(40)
    s.w[1] = 0.0
    s.w[2] = 0.0
    s.w[0] = 1.0
    p = inistate.params_for(s, bc="cont")
    p.tmax = 1e300
    return s, p


@pytest.mark.parametrize("steps", [1, 3, 8, 9, 40])
def test_steps_without_wave_speeds(gpu_lib, steps):
    s, p = gas_at_rest()
    e, o = Engine(p, s.x, s.w), Oracle(p, s.x, s.w)
    e.step(steps)
    o.step(steps)
    assert (e.it, e.t, e.dt) == (o.it, o.t, o.dt) and e.it == steps
    assert same(e.state(), o.state())


def test_server_run_that_finishes_early(gpu_lib):
    """A served run ends at VAC's own tmax = 1e99, which the first dt of gas
    at rest reaches: the steps after it do nothing."""
    s, p = gas_at_rest()
    srv = Server(hbm_budget_bytes=1e9, max_active=2, steps_per_chunk=8)
    st, t, it, _ = srv.result(srv.submit(p, s.x, s.w, 20), wait=60.0)
    p.tmax = 1e99
    o = Oracle(p, s.x, s.w)
    o.step(20)
    assert (it, t) == (o.it, o.t) and same(st, o.state())
    srv.close()


CASES = [
    ("sod", lambda: inistate.sod_1d(64), "minmod", "cont", abi.PREC_FP64),
    ("ot", lambda: inistate.orszag_tang(32), "woodward", "periodic", abi.PREC_FP64),
    ("ot-mixed", lambda: inistate.orszag_tang(48), "minmod", "periodic", abi.PREC_MIXED),
    ("rm-mixed", lambda: inistate.random_modes(24, seed=2, p0=0.5), "woodward", "periodic",
     abi.PREC_MIXED),
]


@pytest.mark.parametrize("name,mk,lim,bc,prec", CASES, ids=[c[0] for c in CASES])
def test_call_lengths_and_stops(gpu_lib, name, mk, lim, bc, prec):
    s = mk()
    p = inistate.params_for(s, limiter=lim, bc=bc, precision=prec)
    ref = Engine(p, s.x, s.w)
    ref.step(43)
    if prec == abi.PREC_FP64:
        o = Oracle(p, s.x, s.w)
        o.step(43)
        assert (ref.it, ref.t) == (o.it, o.t) and same(ref.state(), o.state())
    e = Engine(p, s.x, s.w)
    for n in (0, 1, 2, 7, 9, 8, 16):
        e.step(n)
    assert (e.it, e.t, e.dt) == (43, ref.t, ref.dt) and same(e.state(), ref.state())
    # a save time inside a call, then on to the same end
    e = Engine(p, s.x, s.w)
    assert not e.step(43, tstop=0.4 * ref.t)
    assert 0 < e.it < 43 and e.t >= 0.4 * ref.t
    mid = e.it
    assert not e.step(43 - mid)
    assert (e.it, e.t) == (43, ref.t) and same(e.state(), ref.state())
    # tmax inside a call: the run finishes on the step that reaches it
    p.tmax = 0.4 * ref.t
    e = Engine(p, s.x, s.w)
    assert e.step(400) and e.it == mid
    assert e.step(5) and e.it == mid
