"""A model update after a plan's graphs were captured.

The captured time loops hold the device addresses of the model arrays, so
``fwi2d_update_model`` has to write the new values into the buffers it has
(for VTI: c13, eps and the arrays derived from them too).  Gradients on a
plan that has run before must equal those of a fresh plan on the new model,
bitwise, with other contexts allocating and freeing memory in between.
"""
import numpy as np
import pytest

import oracle as O
import fwi2d_b200 as F
from tests import cases as K

pytestmark = pytest.mark.gpu


def _plan(kind, mc, nx, nz, d, pd, shot):
    P = F.Propagator(0)
    P.set_model(kind, mc, d, d)
    P.set_shots(F.make_params(**pd), [shot])
    return P


@pytest.mark.parametrize("kind", [O.KIND_ELASTIC, O.KIND_VTI])
def test_update_after_capture_equals_fresh_plan(kind):
    nx, nz, d, nt = 96, 64, 0.01, 90
    ma, mb = (K.converted(kind, K.model_case(kind, nx, nz, d, seed=s)) for s in (1, 2))
    sl, rl = K.geometry(nx, nz, d, nr=12)
    pd = K.par_dict(nt=nt, dt=1e-3)
    shot = F.ShotSpec(0, nx, nt, sl[0], sl[1], rl[0], rl[1])
    src = [K.sources(2, nt, 1e-3)]
    obs = [np.random.default_rng(5).normal(size=(2, 12, nt)).astype(np.float32)]
    P1 = _plan(kind, ma, nx, nz, d, pd, shot)
    P1.fwi_gradient(ma, src, obs)
    other = [_plan(kind, ma, nx, nz, d, pd, shot) for _ in range(2)]
    P1.update_model(ma)
    other.pop().close()
    g1, f1 = P1.fwi_gradient(mb, src, obs)
    P2 = _plan(kind, mb, nx, nz, d, pd, shot)
    g2, f2 = P2.fwi_gradient(mb, src, obs)
    for P in [P1, P2] + other:
        P.close()
    assert np.abs(g2).max() > 0
    assert f1 == f2 and np.array_equal(g1, g2)
