"""16-bit snapshots of the acoustic-elastic propagator: the scale of a snapshot
has to cover the interface row, whose uz the coupling sets after the elastic
step, and to stay finite for the first, vanishingly small fields."""
import numpy as np
import pytest

import oracle as O
import fwi2d_b200 as F
from tests import cases as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [3, -1])
def test_ae_gradient_16bit_close_to_fp32(shape):
    nx, nz, d, nt = 90, 60, 0.01, 140
    mc = K.converted(O.KIND_ELASTIC, K.model_case(O.KIND_ELASTIC, nx, nz, d, seed=5))
    oz = 19 * d
    pd = K.par_dict(nt=nt, dt=1e-3, taper=(0, 6, 6, 6), nza=20, acoustic_source=1)
    rx = np.linspace(0.05, 0.84, 20).astype(np.float32)
    shot = F.ShotSpec(0, nx, nt, [0.45], [0.05 + oz], rx, np.full(20, 0.04 + oz, np.float32), water_src_x=[0.453],
                      water_src_z=[0.05], water_rcv_x=rx, water_rcv_z=np.full(20, 0.03, np.float32))
    src = [K.sources(1, nt, 1e-3, f0=25.0, t0=0.03)]
    obs = [np.random.default_rng(2).normal(size=(3, 20, nt)).astype(np.float32)]
    g = {}
    for prec in (F.SNAP_FP32, F.SNAP_FP16, F.SNAP_BF16):
        P = F.Propagator(0)
        P.set_model(O.KIND_AE, mc, d, d, 0.0, oz)
        P.set_shots(F.make_params(**pd, tile_shape=shape, snapshot_precision=prec), [shot])
        g[prec], _ = P.fwi_gradient(mc, src, obs)
        P.close()
    # the storage rounds to 11 and 8 bits; the second time difference of the density term amplifies that
    assert K.rel_l2(g[F.SNAP_FP16], g[F.SNAP_FP32]) < 5e-2
    assert K.rel_l2(g[F.SNAP_BF16], g[F.SNAP_FP32]) < 4e-1
