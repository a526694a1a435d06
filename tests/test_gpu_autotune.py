"""The tile-shape autotuner on gradient plans large enough to be tuned
(>= 2e7 cell-steps) and on grids that the fused time loop does not take (elastic
grids of 32 rows, acoustic shots of 17 to 23 columns): two shots of different record lengths,
tile_shape = -1.

The tuner builds and times candidate plans (sampled forward windows, adjoint
steps, then whole forward + adjoint passes of the close candidates) before it
builds the plan it keeps.  FWI2D_TUNE_CLOSE = 100 sends every shape that fits
through the whole-pass stage, so that stage runs here whatever the sampled
scores, and FWI2D_TUNE_FILE receives the choice, which shows that the tuner ran.
The kept plan must behave exactly like a plan built directly with the chosen
shape: same gradient and misfit, bit for bit; and, since every shape restates
the same operation order, like a plan on another shape too.
"""
import numpy as np
import pytest

import fwi2d_b200 as F
from fwi2d_b200 import workloads as W
from tests import cases as K

pytestmark = pytest.mark.gpu


def _run(kind, tile_shape, nx, nz, nts):
    d, dt = 0.01, 1e-3
    nc = 1 if kind == F.ACOUSTIC else 2
    model = W.convert(kind, K.model_case(kind, nx, nz, d, seed=3))
    shots, srcs, obs = [], [], []
    rng = np.random.default_rng(4)
    for k, nt in enumerate(nts):
        sl, rl = K.geometry(nx, nz, d, nr=12, sx=((0.3 + 0.4 * k) * nx + 0.3) * d)
        shots.append(F.ShotSpec(0, nx, nt, sl[0], sl[1], rl[0], rl[1]))
        srcs.append(K.sources(nc, nt, dt))
        obs.append((rng.standard_normal((nc, 12, nt)) * 1e-3).astype(np.float32))
    assert sum(nx * nz * nt for nt in nts) >= 2e7   # large enough for the tuner
    P = F.Propagator(0)
    P.set_model(kind, model, d, d)
    P.set_shots(F.make_params(**K.par_dict(nt=max(nts), dt=dt, bc=(1, 2, 2, 2), taper=(0, 6, 6, 6)),
                              tile_shape=tile_shape), shots)
    shape = P.plan_info()["tile_shape"]
    g, f = P.fwi_gradient(model, srcs, obs)
    P.close()
    return shape, g, f


@pytest.mark.parametrize("kind,nx,nz,nts,fits", [
    (F.ELASTIC, 420, 32, (900, 660), (2, 3)),
    (F.VTI, 420, 32, (900, 660), (2, 3)),
    (F.ACOUSTIC, 21, 700, (800, 600), (3,)),
])
def test_autotuned_plan_equals_direct_plan(kind, nx, nz, nts, fits, monkeypatch, tmp_path):
    monkeypatch.setenv("FWI2D_TUNE_CLOSE", "100")
    monkeypatch.setenv("FWI2D_TUNE_FILE", str(tmp_path / "tune.txt"))
    shape, g, f = _run(kind, -1, nx, nz, nts)
    assert shape in fits
    assert (tmp_path / "tune.txt").read_text().split()[-1] == str(shape)   # chosen by timing
    shape2, g2, f2 = _run(kind, shape, nx, nz, nts)
    assert shape2 == shape
    assert np.abs(g).max() > 0
    assert np.array_equal(g, g2) and f == f2
    for other in fits:
        _, g3, f3 = _run(kind, other, nx, nz, nts)
        err = K.rel_l2(g, g3)
        print("autotuned shape %d; vs shape %d: gradient rel-L2 %.3e, misfit %.9e vs %.9e" % (shape, other, err, f, f3))
        assert err <= 1e-6
        assert abs(f - f3) <= 1e-6 * abs(f3)
