"""The fused single-kernel sweep of the mixed path (TMA-fed z-marching
tiles): against the FP64 oracle within the mixed tolerance, and against the
split predictor/corrector kernels of the same precision, on periodic,
outflow ('cont') and reflecting ('symm'/'asymm') boundaries and on grids that
are not multiples of the 32x8 tile."""
import os

import numpy as np
import pytest

from oracle.oracle import Oracle
from vac_gb300 import abi, inistate
from vac_gb300.engine import Engine

pytestmark = pytest.mark.gpu

MIXED_REL_L1 = 1e-5     # mixed path vs FP64 oracle, per variable
FUSED_VS_SPLIT = 1e-6   # fused vs split FP32 kernels (different rounding only)


def rel_l1(a, b):
    return [float(np.abs(a[i] - b[i]).sum() / max(np.abs(b[i]).sum(), 1e-300))
            for i in range(a.shape[0])]


def reflecting(p, ndim):
    """symm walls, asymm for the normal momentum (and normal B)."""
    for d in range(ndim):
        for side in (0, 1):
            for iw in range(p.nw):
                p.typeB[2 * d + side][iw] = abi.BC_SYMM
            p.typeB[2 * d + side][1 + d] = abi.BC_ASYMM
            if p.physics == abi.PHYS_MHD:
                p.typeB[2 * d + side][p.ndir + 2 + d] = abi.BC_ASYMM


def _blast(n):
    s = inistate.blast_3d(n)
    return s


CASES = [
    ("rm3-periodic-40", lambda: inistate.random_modes(40, seed=4), "woodward", "periodic", 12, None),
    ("blast3-cont-36", lambda: _blast(36), "woodward", "cont", 10, None),
    ("rm3-reflect-33", lambda: inistate.random_modes(33, seed=5), "minmod", "symm", 8,
     lambda p: reflecting(p, 3)),
    ("hd2-cont-70x50", lambda: _hd(70, 50), "minmod", "cont", 20, None),
    ("ot2-periodic-64", lambda: inistate.orszag_tang(64), "minmod", "periodic", 30, None),
    ("ot2-reflect-45", lambda: inistate.orszag_tang(45), "woodward", "symm", 15,
     lambda p: reflecting(p, 2)),
]


def _hd(nx, ny):
    s = inistate.riemann_2d(8, 11)
    x = inistate.domain_grid((nx, ny), (0.0, 0.0), (1.0, 1.0))
    X, Y = x
    left = X + 0.3 * Y < 0.6
    rho = np.where(left, 1.0, 0.125)
    p = np.where(left, 1.0, 0.1)
    w = inistate.conserve_hd(rho, [np.where(left, 0.2, -0.1), np.zeros_like(X)], p, 1.4)
    s.x, s.w, s.nx = x, w, (nx, ny)
    return s


@pytest.mark.parametrize("name,mk,lim,bc,n,tweak", CASES, ids=[c[0] for c in CASES])
def test_fused_against_oracle_and_split(gpu_lib, monkeypatch, name, mk, lim, bc, n, tweak):
    s = mk()
    p64 = inistate.params_for(s, limiter=lim, bc=bc)
    pm = inistate.params_for(s, limiter=lim, bc=bc, precision=abi.PREC_MIXED)
    if tweak:
        tweak(p64)
        tweak(pm)
    o = Oracle(p64, s.x, s.w)
    o.step(n)
    ref = o.state()
    monkeypatch.setenv("VACGPU_FUSED", "1")
    ef = Engine(pm, s.x, s.w)
    ef.step(n)
    wf = ef.state()
    st = ef.kernel_stats()
    assert st["sweep"][0] > 0, "fused kernel did not run"
    monkeypatch.setenv("VACGPU_FUSED", "0")
    es = Engine(pm, s.x, s.w)
    es.step(n)
    ws = es.state()
    assert es.kernel_stats()["sweep"][0] == 0
    assert max(rel_l1(wf, ref)) <= MIXED_REL_L1, rel_l1(wf, ref)
    assert max(rel_l1(wf, ws)) <= FUSED_VS_SPLIT, rel_l1(wf, ws)


def test_z_chunk_tuning_is_invisible(monkeypatch):
    """At 128^3 the first step call tunes the fused sweep's z chunk from a
    snapshot of the state; the run must be bit-identical to one with the
    chunk pinned (VACGPU_NZC), in state, t and it."""
    s = inistate.random_modes(128, seed=5)
    p = inistate.params_for(s, limiter="woodward", precision=abi.PREC_MIXED)
    tuned = Engine(p, s.x, s.w)
    tuned.step(4)
    monkeypatch.setenv("VACGPU_NZC", "32")
    pinned = Engine(p, s.x, s.w)
    pinned.step(4)
    assert (tuned.it, tuned.t) == (pinned.it, pinned.t)
    assert np.array_equal(tuned.state().view(np.uint64), pinned.state().view(np.uint64))


def test_full_size_conservation_and_symmetry():
    """The benchmark's workload at its full size (256^3 random-mode MHD,
    woodward, periodic, mixed, fused sweeps): without the Powell source the
    flux form conserves mass, momentum, energy and B (volume sums, FP64,
    relative to their scale); and a state mirrored in x evolves into the
    mirror image (m_x and B_x change sign) to FP32 rounding."""
    n = 256
    s = inistate.random_modes(n, seed=0)
    p = inistate.params_for(s, limiter="woodward", precision=abi.PREC_MIXED)
    p.divbfix = 0
    e = Engine(p, s.x, s.w)
    m0 = e.sums()
    e.step(6)
    m1 = e.sums()
    scale = np.abs(s.w).reshape(s.w.shape[0], -1).mean(axis=1)
    assert np.all(np.abs(m1 - m0) <= 2e-7 * np.maximum(scale, 1e-3)), (m1 - m0) / scale
    a = e.state()
    e.close()
    # mirror x -> -x about the box centre: cell i <-> n-1-i
    w = s.w[:, ::-1].copy()
    w[1] = -w[1]
    w[5] = -w[5]
    em = Engine(p, s.x, w)
    em.step(6)
    b = em.state()[:, ::-1]
    em.close()
    b[1] = -b[1]
    b[5] = -b[5]
    rel = [float(np.abs(a[i] - b[i]).sum() / np.abs(a[i]).sum()) for i in range(a.shape[0])]
    assert max(rel) <= 1e-5, rel


def test_full_size_uniform_state_is_preserved_exactly():
    """A uniform state at 256^3 stays bit for bit uniform: identical face
    fluxes cancel exactly and div B is zero."""
    n = 256
    s = inistate.random_modes(n, seed=0)
    w = s.w.copy()
    for iw in range(w.shape[0]):
        w[iw] = w[iw].mean()
    p = inistate.params_for(s, limiter="woodward", precision=abi.PREC_MIXED)
    e = Engine(p, s.x, w)
    e.step(4)
    out = e.state()
    e.close()
    for iw in range(w.shape[0]):
        assert np.all(out[iw] == out[iw].flat[0])
        assert abs(out[iw].flat[0] - np.float32(w[iw].flat[0])) <= 1e-7 * abs(w[iw].flat[0]) + 1e-30


GRAVITY_CASES = [
    ("hd2-gravity-cont", lambda: inistate.riemann_2d(48, 5), "woodward", "cont", 12, [0.0, -0.5]),
    ("ot2-gravity-periodic", lambda: inistate.orszag_tang(40), "minmod", "periodic", 10,
     [0.3, -0.2]),
    ("rm3-gravity-periodic", lambda: inistate.random_modes(20, seed=6), "woodward", "periodic", 6,
     [0.2, 0.0, -0.3]),
]


@pytest.mark.parametrize("name,mk,lim,bc,n,grav", GRAVITY_CASES, ids=[c[0] for c in GRAVITY_CASES])
def test_fused_with_gravity(gpu_lib, monkeypatch, name, mk, lim, bc, n, grav):
    """The fused sweeps' general form (the gravity source of vacusr.gravity.t
    in the predictor and the corrector) against the oracle and the split
    kernels."""
    s = mk()
    p64 = inistate.params_for(s, limiter=lim, bc=bc)
    pm = inistate.params_for(s, limiter=lim, bc=bc, precision=abi.PREC_MIXED)
    o = Oracle(p64, s.x, s.w)
    o.register_source(abi.SRC_GRAVITY, grav)
    o.step(n)
    ref = o.state()
    out = {}
    for fz in ("1", "0"):
        monkeypatch.setenv("VACGPU_FUSED", fz)
        e = Engine(pm, s.x, s.w)
        e.register_source(abi.SRC_GRAVITY, grav)
        e.step(n)
        out[fz] = e.state()
        assert (e.kernel_stats()["sweep"][0] > 0) == (fz == "1")
    assert max(rel_l1(out["1"], ref)) <= MIXED_REL_L1, rel_l1(out["1"], ref)
    assert max(rel_l1(out["1"], out["0"])) <= FUSED_VS_SPLIT, rel_l1(out["1"], out["0"])


def _ot_shape(nx, ny):
    """Orszag-Tang's fields on an nx x ny periodic box (uneven shapes)."""
    x = inistate.domain_grid((nx, ny), (0.0, 0.0), (2 * np.pi, 2 * np.pi))
    X, Y = x
    g = 5.0 / 3.0
    rho = np.full_like(X, g * g)
    v = [-np.sin(Y), np.sin(X)]
    b = [-np.sin(Y), np.sin(2 * X)]
    w = inistate.conserve_mhd(rho, v, np.full_like(X, g), b, g)
    return inistate._snap(x, w, g, True, 2, "Orszag-Tang fields %dx%d" % (nx, ny))


LINE2_SHAPES = [
    ("mhd-61x33-periodic", lambda: _ot_shape(61, 33), "woodward", "periodic", 10, None),
    ("mhd-124x9-periodic", lambda: _ot_shape(124, 9), "minmod", "periodic", 10, None),
    ("mhd-6x70-reflect", lambda: _ot_shape(6, 70), "minmod", "symm", 8,
     lambda p: reflecting(p, 2)),
    ("mhd-129x65-reflect", lambda: _ot_shape(129, 65), "woodward", "symm", 6,
     lambda p: reflecting(p, 2)),
    ("hd-67x131-cont", lambda: _hd(67, 131), "woodward", "cont", 12, None),
    ("hd-128x4-cont", lambda: _hd(128, 4), "minmod", "cont", 12, None),
]


@pytest.mark.parametrize("name,mk,lim,bc,n,tweak", LINE2_SHAPES, ids=[c[0] for c in LINE2_SHAPES])
def test_line_sweep_shapes(gpu_lib, monkeypatch, name, mk, lim, bc, n, tweak):
    """The 2-D line sweep on shapes that cut its 60- and 64-column strips
    and 32-row chunks unevenly (one strip, partly filled strips, fewer rows
    than a chunk, several chunks), against the oracle and the split kernels."""
    test_fused_against_oracle_and_split(gpu_lib, monkeypatch, name, mk, lim, bc, n, tweak)


@pytest.mark.parametrize("nx,lim,bc", [((33, 33, 33), "minmod", "symm"),
                                       ((20, 9, 7), "woodward", "cont"),
                                       ((64, 50, 41), "woodward", "periodic"),
                                       ((97, 88, 90), "minmod", "cont")])
def test_z_chunk_by_size_is_invisible(gpu_lib, monkeypatch, nx, lim, bc):
    """The z chunk that a small grid gets by its size (2 to 8 planes, a last
    chunk of one plane among them) gives the bits of one pinned at 32."""
    s = inistate.random_modes(max(nx), seed=6, p0=0.5)
    s.x = inistate.domain_grid(nx, (0.0,) * 3, tuple(n / max(nx) for n in nx))
    s.w = np.ascontiguousarray(s.w[:, :nx[0], :nx[1], :nx[2]])
    s.nx = nx
    p = inistate.params_for(s, limiter=lim, bc=bc, precision=abi.PREC_MIXED)
    if bc == "symm":
        reflecting(p, 3)
    out = []
    for pin in (None, "32"):
        if pin:
            monkeypatch.setenv("VACGPU_NZC", pin)
        e = Engine(p, s.x, s.w)
        e.step(5)
        assert e.kernel_stats()["sweep"][0] == 15
        out.append((e.t, e.state()))
        e.close()
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1].view(np.uint64), out[1][1].view(np.uint64))



@pytest.mark.parametrize("nx,bc", [((33, 18, 9), "cont"), ((45, 9, 17), "symm"),
                                   ((31, 12, 10), "cont"), ((32, 12, 10), "cont")])
def test_fused_odd_columns(gpu_lib, monkeypatch, nx, bc):
    """MHD on a box cut out of the random modes, whose outflow or reflecting
    x faces carry B_x: with an odd mesh width the last column shares its pair
    with a ghost column."""
    s = inistate.random_modes(max(nx), seed=8, p0=0.5)
    s.x = inistate.domain_grid(nx, (0.0,) * 3, tuple(n / max(nx) for n in nx))
    s.w = np.ascontiguousarray(s.w[:, :nx[0], :nx[1], :nx[2]])
    s.nx = nx
    p = inistate.params_for(s, limiter="minmod", bc=bc, precision=abi.PREC_MIXED)
    if bc == "symm":
        reflecting(p, 3)
    out = []
    for fused in ("1", "0"):
        monkeypatch.setenv("VACGPU_FUSED", fused)
        e = Engine(p, s.x, s.w)
        e.step(1)
        assert (e.kernel_stats()["sweep"][0] > 0) == (fused == "1")
        out.append(e.state())
        e.close()
    assert max(rel_l1(out[0], out[1])) <= FUSED_VS_SPLIT, rel_l1(out[0], out[1])


ROE_CASES = [
    ("rm3-periodic", (40, 33, 36), "woodward", "periodic", {}),
    ("rm3-cont", (33, 18, 9), "minmod", "cont", {}),
    ("rm3-reflect", (30, 20, 17), "woodward", "symm", {}),
    ("rm3-nodivbwave", (31, 16, 24), "minmod", "periodic", {"divbwave": 0}),
    ("rm3-nopowell", (32, 24, 16), "woodward", "periodic", {"divbfix": 0}),
    ("rm2-periodic", (61, 50), "woodward", "periodic", {}),
    ("rm2-cont", (130, 23), "minmod", "cont", {}),
    ("rm2-reflect", (60, 64), "woodward", "symm", {"divbwave": 0}),
]


@pytest.mark.parametrize("name,nx,lim,bc,opt", ROE_CASES, ids=[c[0] for c in ROE_CASES])
def test_fused_roe_against_oracle_and_split(gpu_lib, monkeypatch, name, nx, lim, bc, opt):
    """'tvdmu' on the fused sweeps (ideal MHD, no entropy fix): within the
    mixed tolerance of the FP64 oracle, and within FP32 rounding (twice the
    TVDLF bound: eight waves' products in another order) of the split Roe
    kernels; an entropy fix keeps the split kernels."""
    nd = len(nx)
    s = inistate.random_modes(max(nx), seed=8, p0=0.5, ndim=nd)
    s.x = inistate.domain_grid(nx, (0.0,) * nd, tuple(n / max(nx) for n in nx))
    s.w = np.ascontiguousarray(s.w[(slice(None),) + tuple(slice(0, n) for n in nx)])
    s.nx = nx
    p64 = inistate.params_for(s, limiter=lim, bc=bc)
    pm = inistate.params_for(s, limiter=lim, bc=bc, precision=abi.PREC_MIXED)
    for p in (p64, pm):
        p.typefull = abi.TVDMU
        for k, v in opt.items():
            setattr(p, k, v)
        if bc == "symm":
            reflecting(p, nd)
    # two steps against the walls: the oracle's pressure is negative after four
    n = 2 if bc == "symm" else 8
    o = Oracle(p64, s.x, s.w)
    o.step(n)
    out = []
    for fused in ("1", "0"):
        monkeypatch.setenv("VACGPU_FUSED", fused)
        e = Engine(pm, s.x, s.w)
        e.step(n)
        assert (e.kernel_stats()["sweep"][0] > 0) == (fused == "1")
        assert abs(e.t - o.t) <= 1e-6 * o.t
        out.append(e.state())
        assert max(rel_l1(out[-1], o.state())) <= MIXED_REL_L1
        assert e.nerror() == o.nerror()
        e.close()
    assert max(rel_l1(out[0], out[1])) <= 2 * FUSED_VS_SPLIT
    monkeypatch.setenv("VACGPU_FUSED", "1")
    pm.typeentropy[0] = abi.ENTROPY_HARTEN
    e = Engine(pm, s.x, s.w)
    e.step(2)
    assert e.kernel_stats()["sweep"][0] == 0


def _hd3(nx, seed=8):
    """Gas with the random modes' density and velocity on a box of cubic cells."""
    s = inistate.random_modes(max(nx), seed=seed, p0=0.5)
    w = s.w[(slice(0, 4),) + tuple(slice(0, n) for n in nx)]
    x = inistate.domain_grid(nx, (0.0,) * 3, tuple(n / max(nx) for n in nx))
    w = inistate.conserve_hd(w[0], [w[1 + d] / w[0] for d in range(3)],
                             np.full(nx, 0.5), 1.4)
    return inistate._snap(x, w, 1.4, False, 3, "random-mode gas")


HD3_CASES = [
    ("hd3-33x18x9-cont", (33, 18, 9), "woodward", "cont"),
    ("hd3-45x9x17-reflect", (45, 9, 17), "minmod", "symm"),
    ("hd3-31x12x10-cont", (31, 12, 10), "minmod", "cont"),
    ("hd3-32x12x10-reflect", (32, 12, 10), "woodward", "symm"),
    ("hd3-32x24x30-cont", (32, 24, 30), "woodward", "cont"),
    ("hd3-65x20x11-periodic", (65, 20, 11), "woodward", "periodic"),
    ("hd3-64x33x36-periodic", (64, 33, 36), "minmod", "periodic"),
]


@pytest.mark.parametrize("name,nx,lim,bc", HD3_CASES, ids=[c[0] for c in HD3_CASES])
def test_fused_gas_3d(gpu_lib, monkeypatch, name, nx, lim, bc):
    """3-D gas on the pair sweep, whose cells carry five variables where MHD's
    carry eight: odd and even widths, each kind of face."""
    test_fused_against_oracle_and_split(
        gpu_lib, monkeypatch, name, lambda: _hd3(nx), lim, bc, 8,
        (lambda p: reflecting(p, 3)) if bc == "symm" else None)


LONG_ITEMS = [
    # items of 2 rows and a last one of one row; of 4 and one; of 16 and 13
    ("mhd-600x131-reflect", lambda: _ot_shape(600, 131), "minmod", "symm", 4,
     lambda p: reflecting(p, 2)),
    ("hd-700x777-cont", lambda: _hd(700, 777), "woodward", "cont", 3, None),
    ("mhd-1210x1101-periodic", lambda: _ot_shape(1210, 1101), "woodward", "periodic", 2, None),
]


@pytest.mark.parametrize("name,mk,lim,bc,n,tweak", LONG_ITEMS, ids=[c[0] for c in LONG_ITEMS])
def test_line_sweep_items_of_several_rows(gpu_lib, monkeypatch, name, mk, lim, bc, n, tweak):
    """2-D grids with more rows than warps, whose work items march several
    rows (the shapes above have items of one row) and end on a shorter item,
    against the oracle and the split kernels."""
    test_fused_against_oracle_and_split(gpu_lib, monkeypatch, name, mk, lim, bc, n, tweak)


@pytest.mark.parametrize("nx,lim,bc", [((600, 131), "woodward", "cont"),
                                       ((600, 131), "minmod", "symm"),
                                       ((601, 400), "minmod", "periodic")])
def test_line_sweep_roe_items_of_several_rows(gpu_lib, monkeypatch, nx, lim, bc):
    test_fused_roe_against_oracle_and_split(gpu_lib, monkeypatch, "rows", nx, lim, bc, {})


@pytest.mark.parametrize("lim", ["minmod", "woodward"])
@pytest.mark.parametrize("roe", [False, True])
def test_rows_per_item_are_invisible(gpu_lib, roe, lim):
    """A periodic 61x50 state repeated along y: 26 copies run in items of three
    rows, one copy in items of one, and each copy keeps the bits.  (Cells of
    1/64, so that every cell width is exact at either height.)"""
    s = inistate.random_modes(64, seed=9, p0=0.5, ndim=2)
    w = s.w[:, :61, :50]
    out = []
    for k in (1, 26):
        x = np.stack(np.meshgrid((np.arange(61) + 0.5) / 64, (np.arange(50 * k) + 0.5) / 64,
                                 indexing="ij"))
        t = inistate._snap(x, np.ascontiguousarray(np.tile(w, (1, 1, k))), 5.0 / 3.0, True, 2,
                           "repeated modes")
        p = inistate.params_for(t, limiter=lim, precision=abi.PREC_MIXED)
        if roe:
            p.typefull = abi.TVDMU
        e = Engine(p, t.x, t.w)
        e.step(6)
        assert e.kernel_stats()["sweep"][0] == 12
        out.append((e.t, e.state()))
        e.close()
    assert out[0][0] == out[1][0]
    many = np.ascontiguousarray(np.tile(out[0][1], (1, 1, 26)))
    assert np.array_equal(many.view(np.uint64), out[1][1].view(np.uint64))


@pytest.mark.parametrize("nx,lim,bc", [((33, 33, 33), "minmod", "symm"),
                                       ((64, 50, 41), "woodward", "periodic"),
                                       ((97, 88, 90), "minmod", "cont")])
def test_z_chunk_of_roe_sweeps_is_invisible(gpu_lib, monkeypatch, nx, lim, bc):
    s = inistate.random_modes(max(nx), seed=6, p0=0.5)
    s.x = inistate.domain_grid(nx, (0.0,) * 3, tuple(n / max(nx) for n in nx))
    s.w = np.ascontiguousarray(s.w[:, :nx[0], :nx[1], :nx[2]])
    s.nx = nx
    p = inistate.params_for(s, limiter=lim, bc=bc, precision=abi.PREC_MIXED)
    p.typefull = abi.TVDMU
    if bc == "symm":
        reflecting(p, 3)
    n = 2 if bc == "symm" else 5
    out = []
    for pin in (None, "5", "32"):
        if pin:
            monkeypatch.setenv("VACGPU_NZC", pin)
        e = Engine(p, s.x, s.w)
        e.step(n)
        assert e.kernel_stats()["sweep"][0] == 3 * n
        out.append((e.t, e.state()))
        e.close()
    for t, w in out[1:]:
        assert t == out[0][0] and np.array_equal(w.view(np.uint64), out[0][1].view(np.uint64))


ROE_FORMS = [
    ("rm3-stretched", (24, 33, 18), "woodward", "stretched"),
    ("rm2-stretched", (70, 50), "minmod", "stretched"),
    ("rm3-gravity", (24, 33, 18), "minmod", "gravity"),
    ("rm2-gravity", (70, 50), "woodward", "gravity"),
]


@pytest.mark.parametrize("name,nx,lim,form", ROE_FORMS, ids=[c[0] for c in ROE_FORMS])
def test_fused_roe_on_stretched_grids_and_with_gravity(gpu_lib, monkeypatch, name, nx, lim, form):
    """The fused Roe flux takes |a| without the factor dt*2/(dx(i)+dx(j)) that
    the split kernels multiply by and divide out again: on cells whose widths
    vary, and with the gravity source, against the oracle and the split
    kernels (bounds as for the other Roe cases)."""
    nd = len(nx)
    s = inistate.random_modes(max(nx), seed=8, p0=0.5, ndim=nd)
    s.x = inistate.domain_grid(nx, (0.0,) * nd, tuple(n / max(nx) for n in nx))
    s.w = np.ascontiguousarray(s.w[(slice(None),) + tuple(slice(0, n) for n in nx)])
    s.nx = nx
    if form == "stretched":
        s = inistate.stretched(s)
    p64 = inistate.params_for(s, limiter=lim)
    pm = inistate.params_for(s, limiter=lim, precision=abi.PREC_MIXED)
    p64.typefull = pm.typefull = abi.TVDMU
    g = [0.3, -0.2, 0.1][:nd]
    o = Oracle(p64, s.x, s.w)
    if form == "gravity":
        o.register_source(abi.SRC_GRAVITY, g)
    o.step(8)
    out = []
    for fused in ("1", "0"):
        monkeypatch.setenv("VACGPU_FUSED", fused)
        e = Engine(pm, s.x, s.w)
        if form == "gravity":
            e.register_source(abi.SRC_GRAVITY, g)
        e.step(8)
        assert (e.kernel_stats()["sweep"][0] > 0) == (fused == "1")
        assert abs(e.t - o.t) <= 1e-6 * o.t
        out.append(e.state())
        assert max(rel_l1(out[-1], o.state())) <= MIXED_REL_L1
        e.close()
    assert max(rel_l1(out[0], out[1])) <= 2 * FUSED_VS_SPLIT


def _superbee(nx, bc, mhd=True):
    s = inistate.random_modes(max(nx), seed=6, p0=0.5)
    s.x = inistate.domain_grid(nx, (0.0,) * 3, tuple(n / max(nx) for n in nx))
    s.w = np.ascontiguousarray(s.w[:, :nx[0], :nx[1], :nx[2]])
    s.nx = nx
    if not mhd:
        s = _hd3(nx, seed=6)
    return s, inistate.params_for(s, limiter="superbee", bc=bc, precision=abi.PREC_MIXED)


@pytest.mark.parametrize("nx,bc,mhd", [((33, 17, 33), "cont", True), ((64, 50, 41), "periodic", True),
                                       ((31, 20, 9), "cont", False),
                                       ((97, 88, 90), "periodic", False)])
def test_z_chunk_of_the_one_cell_kernel_is_invisible(gpu_lib, monkeypatch, nx, bc, mhd):
    """Limiters without a pair kernel: the chunk that a grid gets by its size
    gives the bits of one pinned at 32."""
    s, p = _superbee(nx, bc, mhd)
    out = []
    for pin in (None, "32"):
        if pin:
            monkeypatch.setenv("VACGPU_NZC", pin)
        e = Engine(p, s.x, s.w)
        e.step(4)
        assert e.kernel_stats()["sweep"][0] == 12
        out.append((e.t, e.state()))
        e.close()
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1].view(np.uint64), out[1][1].view(np.uint64))


def test_z_chunk_of_the_one_cell_kernel_fits_the_grid(gpu_lib, monkeypatch):
    """At 130x127x133 the size's chunk is no slower than the better of 8 and
    16 planes by more than a tenth (32 planes: by 30 to 40 %)."""
    s, p = _superbee((130, 127, 133), "cont")
    us = {}
    for pin in (None, "8", "16"):
        if pin:
            monkeypatch.setenv("VACGPU_NZC", pin)
        e = Engine(p, s.x, s.w)
        e.step(4)
        for _ in range(3):
            e.timing(True)
            e.step(6)
            n, ms = e.kernel_stats()["sweep"]
            us[pin] = min(us.get(pin, 1e9), 1e3 * ms / n)
        e.timing(False)
        e.close()
    assert us[None] <= 1.1 * min(us["8"], us["16"]), us
