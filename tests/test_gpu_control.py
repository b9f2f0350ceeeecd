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


# cells of the speed checks and their steps: a launch-bound grid
N_DUST, STEPS_DUST = 64, 400


def dust_and_gas():
    """Pressureless gas that flows along x (no wave speed along y, so each
    step's dt needs the cell-centred pass) and ordinary gas on one grid."""
    from tests.test_gpu_skipped_steps import dust
    return dust(N_DUST, N_DUST), inistate.riemann_2d(N_DUST, 3)


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
def test_passes_at_every_step_cost_their_launches(gpu_lib, prec):
    """Steps that need the cell-centred passes cost six launches more than
    others, not a round trip to the host each: no more than 40 us a step, and
    a served run no more than a run alone, its set-up and one more chunk."""
    import time
    sd, sg = dust_and_gas()
    best, eng = {}, {}
    for name, s in (("dust", sd), ("gas", sg)):
        e = eng[name] = Engine(inistate.params_for(s, precision=prec), s.x, s.w)
        for _ in range(4):
            e.upload(s.w)
            t0 = time.perf_counter()
            e.step(STEPS_DUST)
            best[name] = min(best.get(name, 1e9), time.perf_counter() - t0)
            assert e.it == STEPS_DUST
    assert best["dust"] - best["gas"] <= 40e-6 * STEPS_DUST, best
    p = inistate.params_for(sd, precision=prec)
    srv = Server(hbm_budget_bytes=1e9, max_active=2, steps_per_chunk=16)
    t0 = time.perf_counter()
    st, t, it, tts = srv.result(srv.submit(p, sd.x, sd.w, STEPS_DUST), wait=120.0)
    served = time.perf_counter() - t0
    srv.close()
    assert it == STEPS_DUST and t == eng["dust"].t and same(st, eng["dust"].state())
    assert served <= 2 * best["dust"] + 0.05, (served, best)
    if prec == abi.PREC_FP64:
        o = Oracle(p, sd.x, sd.w)
        o.step(STEPS_DUST)
        assert t == o.t and same(st, o.state())


@pytest.mark.parametrize("chunk", [1, 7, 16])
def test_served_gas_that_stalls_late(gpu_lib, chunk):
    """Wave speeds along y that die out (the gas that moved along y leaves
    through an outflow face; below 1e-99 a speed sets no dt): the passes are
    needed from the middle of the run on."""
    from tests.test_gpu_skipped_steps import dust
    s = dust(12, 9)
    s.w[2, -1, :] = 1e-80 * s.w[0, -1, :]
    p = inistate.params_for(s, bc="cont")
    o = Oracle(p, s.x, s.w)
    o.step(20)
    assert np.abs(o.state()[2]).max() > 1e-97
    o.step(40)
    assert np.abs(o.state()[2]).max() < 1e-101
    srv = Server(hbm_budget_bytes=1e9, max_active=2, steps_per_chunk=chunk)
    st, t, it, _ = srv.result(srv.submit(p, s.x, s.w, 60), wait=60.0)
    srv.close()
    assert (it, t) == (60, o.t) and same(st, o.state())
    e = Engine(p, s.x, s.w)
    for n in (1, 2, 30, 27):
        e.step(n)
    assert (e.it, e.t) == (60, o.t) and same(e.state(), o.state())
