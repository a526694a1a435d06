"""The fused time loop (all steps of a pass in one launch of resident CTAs that
meet between steps) against the oracle and the tile kernel.

Grids sit at the edges of its units: the smallest it takes (40 rows, 16
columns), one cell either side of a full interior window (32 x 16 from row 4
and column 6), partial last windows and band units, z windows that end flush.
Every result restates the reference's FP32 operations, so traces, snapshots
and gradients must equal the oracle's bit for bit.
"""
import numpy as np
import pytest

import oracle as O
import fwi2d_b200 as F
from tests import cases as K
from tests.test_gpu_parity import run_gpu

pytestmark = pytest.mark.gpu


def fused_shape():
    return F.load().fwi2d_tile_shape_count() - 1


@pytest.mark.parametrize("kind,mt,bc", [
    (O.KIND_ELASTIC, 0, (1, 2, 2, 2)),
    (O.KIND_ELASTIC, 1, (2, 2, 2, 2)),
    (O.KIND_ELASTIC, 0, (1, 1, 1, 1)),
    (O.KIND_VTI, 0, (1, 2, 2, 2)),
    (O.KIND_VTI, 1, (2, 1, 2, 1)),
])
@pytest.mark.parametrize("grid", [(16, 40), (17, 41), (28, 42), (29, 43), (44, 74), (45, 75), (61, 107), (120, 200)])
def test_fused_vs_oracle(kind, mt, bc, grid):
    nx, nz = grid
    d, nt = 0.01, 150
    mc = K.converted(kind, K.model_case(kind, nx, nz, d, seed=3))
    sl, rl = K.geometry(nx, nz, d, nr=14)
    # sources and receivers in the bands, on their seams and in the interior windows
    sl = (np.array([0.05, 0.3 * nx * d, (nx - 7.2) * d], np.float32), np.array([0.02, 0.055, 0.36], np.float32))
    rz = np.array([0.02, 0.045, 0.055, 0.065, 0.2, 0.35, (nz - 7.3) * d, (nz - 6.2) * d, (nz - 2.4) * d], np.float32)
    rl = (np.linspace(1.2 * d, (nx - 2.3) * d, 27).astype(np.float32), np.tile(rz, 3))
    pd = K.par_dict(nt=nt, dt=1e-3, bc=bc, mt=mt, taper=(0, 6, 5, 6))
    ns = len(sl[0])
    src = np.repeat(K.sources(3 if mt else 2, nt, 1e-3, f0=25.0, t0=0.03), ns, axis=1)
    port = O.Port(32)
    par = O.make_par(**pd, ns=ns, nr=len(rl[0]))
    rcv_o, full_o = K.oracle_forward(port, kind, mc, src, par, nx, nz, d, sl, rl, mt=mt)
    adj = np.ascontiguousarray(rcv_o[:, :, ::-1])
    g_o = np.zeros((5 if kind == O.KIND_VTI else 3, nx, nz), np.float32)
    srcb = np.zeros((3 if mt else 2, ns, nt), np.float32)
    port.propagate(kind, 1, mc, adj, srcb, par, nx, nz, d, d, 0.0, 0.0, rl, sl, inj_type=0, full=full_o, grad=g_o)
    rcv_g, g_g, snaps = run_gpu(kind, mc, src, pd, nx, nz, d, sl, rl, adj_src=adj, mt=mt, shape=fused_shape())
    step = max(1, nt // 5)
    want = np.stack([full_o[k] for k in range(0, nt, step)])
    print("fused kind %d mt %d bc %s grid %s: traces %.4f snapshots %.4f gradient %.4f equal" % (
        kind, mt, bc, grid, np.mean(rcv_g == rcv_o), np.mean(snaps == want), np.mean(g_g == g_o[:3])))
    assert np.abs(g_o).max() > 0
    assert np.array_equal(rcv_g, rcv_o)
    assert np.array_equal(snaps, want)
    assert np.array_equal(g_g, g_o[:3])


def _gradient(kind, shape, prec, every, compensated, nx=150, nz=75, nt=97):
    d = 0.01
    base = O.KIND_ELASTIC if kind == O.KIND_AE else kind
    mc = K.converted(base, K.model_case(base, nx, nz, d, seed=5))
    rng = np.random.default_rng(9)
    oz = 0.0
    pd = K.par_dict(nt=nt, dt=1e-3, taper=(0, 6, 6, 6))
    if kind == O.KIND_AE:
        pd.update(nza=20, acoustic_source=1)
        oz = 19 * d
    shots, src, obs = [], [], []
    for x0, w, n in ((0, 150, nt), (3, 61, nt), (70, 77, nt)) if every else ((0, 150, nt), (3, 61, nt - 31), (70, 77, nt - 10)):
        rx = ((x0 + np.linspace(2.2, w - 3.3, 11)) * d).astype(np.float32)
        sx, sz = [(x0 + 0.5 * w) * d], [0.06]
        rz = np.full(11, 0.04, np.float32)
        kw = {}
        if kind == O.KIND_AE:
            kw = dict(water_src_x=sx, water_src_z=[0.05], water_rcv_x=rx, water_rcv_z=np.full(11, 0.03, np.float32))
        shots.append(F.ShotSpec(x0, w, n, sx, [sz[0] + oz], rx, rz + np.float32(oz), **kw))
        ns = 1 if kind in (O.KIND_AE, O.KIND_ACOUSTIC) else 2
        nc = {O.KIND_AE: 3, O.KIND_ACOUSTIC: 1}.get(kind, 2)
        src.append(K.sources(ns, n, 1e-3, f0=25.0, t0=0.03).reshape(ns, 1, n))
        obs.append(rng.normal(size=(nc, 11, n)).astype(np.float32))
    P = F.Propagator(0)
    P.set_model(kind, mc, d, d, 0.0, oz)
    P.set_shots(F.make_params(**pd, tile_shape=shape, snapshot_precision=prec, checkpoint_every=every,
                              compensated=compensated), shots)
    out = [P.fwi_gradient(mc, src, obs) for _ in range(2)]
    rcv = P.forward(src, store=False)
    P.close()
    return out, rcv


@pytest.mark.parametrize("kind", [O.KIND_ELASTIC, O.KIND_VTI, O.KIND_AE, O.KIND_ACOUSTIC])
@pytest.mark.parametrize("prec,every,compensated", [(0, 0, 0), (2, 0, 1), (1, 20, 0), (0, 7, 1)])
def test_fused_plan_equals_tile_plan(kind, prec, every, compensated):
    """Uneven windows and records, 16-bit snapshots, replayed segments and
    compensated accumulation: the loop is cut into several launches there."""
    if kind == O.KIND_AE and every:
        pytest.skip("checkpoint-and-recompute is not available for the acoustic-elastic propagator")
    a, ra = _gradient(kind, fused_shape(), prec, every, compensated)
    b, rb = _gradient(kind, 3, prec, every, compensated)
    for (ga, fa), (gb, fb) in zip(a, b):
        assert np.abs(gb).max() > 0
        assert fa == fb and np.array_equal(ga, gb)
    for x, y in zip(ra, rb):
        assert np.array_equal(x, y)


def _imaging(kind, shape, prec, sub, nt=61):
    """Forward and adjoint imaging on one context, first with a snapshot every
    step, whose values stay in the CTAs' shared memory, then with every sub-th."""
    nx, nz, d = 61, 107, 0.01
    base = O.KIND_ELASTIC if kind == O.KIND_AE else kind
    mc = K.converted(base, K.model_case(base, nx, nz, d, seed=5))
    oz = 19 * d if kind == O.KIND_AE else 0.0
    rx, rz = np.linspace(0.05, 0.55, 11).astype(np.float32), np.full(11, 0.04, np.float32)
    kw = {}
    if kind == O.KIND_AE:
        kw = dict(water_src_x=[0.303], water_src_z=[0.12], water_rcv_x=rx, water_rcv_z=rz)
    shot = F.ShotSpec(0, nx, nt, [0.303], [0.3 + oz], rx, rz + np.float32(oz), **kw)
    ns = 1 if kind in (O.KIND_AE, O.KIND_ACOUSTIC) else 2
    nc = {O.KIND_AE: 3, O.KIND_ACOUSTIC: 1}.get(kind, 2)
    src = [K.sources(ns, nt, 1e-3, f0=25.0, t0=0.03).reshape(ns, 1, nt)]
    adj = [np.random.default_rng(9).normal(size=(nc, 11, nt)).astype(np.float32)]
    P = F.Propagator(0)
    P.set_model(kind, mc, d, d, 0.0, oz)
    for every in (1, sub):
        pd = K.par_dict(nt=nt, dt=1e-3, taper=(0, 6, 6, 6), sub=every)
        if kind == O.KIND_AE:
            pd.update(nza=20, acoustic_source=1)
        P.set_shots(F.make_params(**pd, tile_shape=shape, snapshot_precision=prec), [shot])
        P.forward(src, store=True)
        g = P.adjoint(adj)
    P.close()
    return g


@pytest.mark.parametrize("kind", [O.KIND_ELASTIC, O.KIND_VTI, O.KIND_AE, O.KIND_ACOUSTIC])
@pytest.mark.parametrize("prec,sub", [(0, 2), (0, 7), (0, 59), (0, 60), (0, 62), (2, 3), (2, 100), (1, 63)])
def test_fused_subsampled_imaging_equals_tile_plan(kind, prec, sub):
    """Snapshots every sub steps of 61 samples, up to one snapshot only (sub
    beyond the record: the first is the last, and none follows it)."""
    a, b = _imaging(kind, fused_shape(), prec, sub), _imaging(kind, 3, prec, sub)
    assert np.array_equal(a, b)
    if kind in (O.KIND_ELASTIC, O.KIND_VTI):
        assert (np.abs(b).max() > 0) == (sub < 62)   # the field at time 0 is zero


@pytest.mark.parametrize("bc", [(1, 2, 2, 2), (3, 1, 2, 3)])
@pytest.mark.parametrize("grid", [(24, 40), (40, 47), (61, 107), (150, 210)])
def test_acoustic_loop_vs_oracle(bc, grid):
    """The acoustic time loop: tiles of the closures only, and z-pair windows."""
    nx, nz = grid
    kind, d, nt = O.KIND_ACOUSTIC, 0.01, 150
    mc = K.converted(kind, K.model_case(kind, nx, nz, d, seed=3))
    sl, rl = K.geometry(nx, nz, d, nr=14, sz=0.2)
    pd = K.par_dict(nt=nt, dt=1e-3, bc=bc, taper=(0, 6, 5, 6))
    src = K.sources(1, nt, 1e-3, f0=25.0, t0=0.03)
    port = O.Port(32)
    par = O.make_par(**pd, ns=1, nr=14)
    rcv_o, full_o = K.oracle_forward(port, kind, mc, src, par, nx, nz, d, sl, rl)
    adj = np.ascontiguousarray(rcv_o[:, :, ::-1])
    g_o = K.oracle_adjoint(port, kind, mc, adj, par, nx, nz, d, sl, rl, full_o)
    rcv_g, g_g, _ = run_gpu(kind, mc, src, pd, nx, nz, d, sl, rl, adj_src=adj, shape=fused_shape())
    assert np.abs(g_o).max() > 0
    assert np.array_equal(rcv_g, rcv_o)
    assert np.array_equal(g_g, g_o)


def test_fused_wait_limit_returns_timeout(monkeypatch):
    """A meeting of the CTAs that reaches its poll limit (0 here, so at once; the
    second bound is the ordinary one and nothing is left waiting) is reported,
    and the context stays usable."""
    kind, nx, nz, d, nt = O.KIND_ELASTIC, 60, 50, 0.01, 60
    mc = K.converted(kind, K.model_case(kind, nx, nz, d, seed=11))
    sl, rl = K.geometry(nx, nz, d, nr=8)
    pd = K.par_dict(nt=nt, dt=1e-3)
    src = [K.sources(2, nt, 1e-3)]
    P = F.Propagator(0)
    P.set_model(kind, mc, d, d)
    shot = F.ShotSpec(0, nx, nt, sl[0], sl[1], rl[0], rl[1])
    monkeypatch.setenv("FWI2D_SPIN_LIMIT", "0")
    P.set_shots(F.make_params(**pd, tile_shape=fused_shape()), [shot])
    with pytest.raises(F.Fwi2dError, match="reached its limit"):
        P.forward(src, store=True)
    with pytest.raises(F.Fwi2dError):
        P.adjoint([np.zeros((2, 8, nt), np.float32)])
    monkeypatch.delenv("FWI2D_SPIN_LIMIT")
    out = []
    for shape in (fused_shape(), 3):
        P.set_shots(F.make_params(**pd, tile_shape=shape), [shot])
        out.append(P.forward(src, store=False)[0])
    P.close()
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("kind,shape,nt,every,compensated,adjoint", [
    (O.KIND_ELASTIC, -1, 97, 0, 1, 1 + 12 + 12 + 1 + 1),       # 12 windows of 8 steps
    (O.KIND_ELASTIC, -1, 100, 0, 1, 1 + 13 + 12 + 1 + 1),      # and one of 3
    (O.KIND_ELASTIC, -1, 97, 20, 1, None),                     # cut by windows and by segments
    (O.KIND_ACOUSTIC, -1, 60, 7, 1, None),
    (O.KIND_ELASTIC, -1, 60, 1, 0, None),                      # a segment a step: its first forward run is empty
    (O.KIND_ELASTIC, -1, 60, 0, 0, 1 + 1 + 1),
    (O.KIND_AE, -1, 60, 0, 1, None),
    (O.KIND_ELASTIC, 3, 97, 0, 1, 1 + 96 + 12 + 1 + 1),
    (O.KIND_ELASTIC, 14, 60, 7, 1, None),
    (O.KIND_ACOUSTIC, 3, 60, 7, 0, None),
])
def test_plan_info_counts_the_launches(kind, shape, nt, every, compensated, adjoint):
    """The counts of a plan that has not run are those its passes then capture
    (init, steps, flushes, final flush, scatter of one shot)."""
    nx, nz, d = 60, 64, 0.01
    base = O.KIND_ELASTIC if kind == O.KIND_AE else kind
    mc = K.converted(base, K.model_case(base, nx, nz, d, seed=11))
    oz = 19 * d if kind == O.KIND_AE else 0.0
    sl, rl = K.geometry(nx, nz, d, nr=8, sz=0.2)
    pd = K.par_dict(nt=nt, dt=1e-3)
    kw = {}
    if kind == O.KIND_AE:
        pd.update(nza=20, acoustic_source=0)
        kw = dict(water_rcv_x=rl[0], water_rcv_z=rl[1])
    P = F.Propagator(0)
    P.set_model(kind, mc, d, d, 0.0, oz)
    P.set_shots(F.make_params(**pd, tile_shape=shape, checkpoint_every=every, compensated=compensated),
                [F.ShotSpec(0, nx, nt, sl[0], sl[1] + np.float32(oz), rl[0], rl[1] + np.float32(oz), **kw)])
    before = P.plan_info()
    rcv = P.forward([K.sources(P.ncomp(), nt, 1e-3)], store=True)
    P.adjoint(rcv)
    after = P.plan_info()
    P.close()
    assert before == after
    assert adjoint is None or after["launches_adjoint"] == adjoint


def _spots(limit, per, pivots, corner, over):
    """Points whose 3 x 3 footprints put exactly `limit` entries (beyond it: two
    corner ones more) into one unit: `per` entries a point inside it, one cell's
    for each point around `corner`."""
    n = limit // (9 * per)
    k = (limit - n * 9 * per) // per + 2 * over
    pts = [pivots[i % len(pivots)] for i in range(n)] + [corner] * k
    return [(x + 0.3 - 0.011 * i % 0.5, z + 0.2 - 0.007 * i % 0.4) for i, (x, z) in enumerate(pts)]


@pytest.mark.parametrize("kind,mt", [(O.KIND_ELASTIC, 0), (O.KIND_ELASTIC, 1), (O.KIND_VTI, 0), (O.KIND_ACOUSTIC, 0)])
@pytest.mark.parametrize("over", [0, 1, 30])
def test_fused_dense_arrays_vs_oracle(kind, mt, over):
    """As many injection entries as a unit stages, and more: windows 256, bands 512
    in the adjoint and 256 in the forward, acoustic tiles 512."""
    nx, nz, d, nt = 45, 75, 0.01, 60
    mc = K.converted(kind, K.model_case(kind, nx, nz, d, seed=3))
    if kind == O.KIND_ACOUSTIC:
        inner = [(x, z) for x in range(2, 14) for z in range(2, 30, 3)]
        s = r = _spots(512, 1, inner, (16, 32), over)
    else:
        window = [(x, z) for x in range(24, 36, 2) for z in range(38, 64, 3)]   # cells 22..37, 36..67
        band = [(x, z) for x in range(1, 5) for z in range(1, 23)]           # cells 0..5, 0..24
        top = [(x, 2) for x in range(8, 32)]                                 # cells 6..33, 0..5
        s = (_spots(256, 2, window, (38, 68), over) + _spots(256, 2, band, (6, 25), over) +
             _spots(256, 2, top, (34, 6), over))
        r = (_spots(256, 2, window, (38, 68), over) + _spots(512, 2, band, (6, 25), over) +
             _spots(512, 2, top, (34, 6), over))
    sl, rl = (tuple(np.array([p[c] * d for p in q], np.float32) for c in (0, 1)) for q in (s, r))
    pd = K.par_dict(nt=nt, dt=1e-3, mt=mt, taper=(0, 6, 5, 6))
    nc = 1 if kind == O.KIND_ACOUSTIC else (3 if mt else 2)
    src = np.repeat(K.sources(nc, nt, 1e-3, f0=25.0, t0=0.03), len(s), axis=1)
    src = (src * np.random.default_rng(2).normal(size=(1, len(s), 1))).astype(np.float32)
    port = O.Port(32)
    par = O.make_par(**pd, ns=len(s), nr=len(r))
    rcv_o, full_o = K.oracle_forward(port, kind, mc, src, par, nx, nz, d, sl, rl, mt=mt)
    adj = np.ascontiguousarray(rcv_o[:, :, ::-1])
    ng = 5 if kind == O.KIND_VTI else (2 if kind == O.KIND_ACOUSTIC else 3)
    g_o = np.zeros((ng, nx, nz), np.float32)
    port.propagate(kind, 1, mc, adj, np.zeros((nc, len(s), nt), np.float32), par, nx, nz, d, d, 0.0, 0.0, rl, sl,
                   inj_type=0, full=full_o, grad=g_o)
    rcv_g, g_g, _ = run_gpu(kind, mc, src, pd, nx, nz, d, sl, rl, adj_src=adj, mt=mt, shape=fused_shape())
    assert np.abs(g_o).max() > 0
    assert np.array_equal(rcv_g, rcv_o)
    assert np.array_equal(g_g, g_o[:3])


def test_two_contexts_run_their_loops_at_once():
    """Two threads, a context and a stream each, both with more units than the GPU
    holds CTAs: a cooperative launch starts with all of its CTAs or waits, so
    neither loop starves the other, and results are those of each alone."""
    import threading
    nx, nz, d, nt = 400, 300, 0.01, 150
    jobs = []
    for k, kind in enumerate((O.KIND_ELASTIC, O.KIND_ACOUSTIC)):
        mc = K.converted(kind, K.model_case(kind, nx, nz, d, seed=3 + k))
        sl, rl = K.geometry(nx, nz, d, nr=20)
        P = F.Propagator(0)
        P.set_model(kind, mc, d, d)
        P.set_shots(F.make_params(**K.par_dict(nt=nt, dt=1e-3)), [F.ShotSpec(0, nx, nt, sl[0], sl[1], rl[0], rl[1])] * 2)
        src = [K.sources(P.ncomp(), nt, 1e-3)] * 2
        obs = [np.zeros((P.ncomp(), 20, nt), np.float32)] * 2
        jobs.append((P, mc, src, obs, P.fwi_gradient(mc, src, obs)))
    bad = []

    def work(P, mc, src, obs, want):
        for _ in range(8):
            g, f = P.fwi_gradient(mc, src, obs)
            if f != want[1] or not np.array_equal(g, want[0]):
                bad.append(f)
    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for j in jobs:
        j[0].close()
    assert not bad
