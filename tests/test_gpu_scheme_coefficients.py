"""RUNGKU coefficients other than the reference's, in the FMA build, where Z of
stage 2 may be formed from U1 and U0: a scheme whose ZETA1 exceeds GAM1, down
to GAM1 = 0, is stepped as well as the reference's own."""
import numpy as np
import pytest

from test_gpu_parity import FAST_TOL, _cfg, _fields, _gpu_or_skip, _random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmag,lrot", [(1, 1), (1, 0), (0, 1), (0, 0)])
@pytest.mark.parametrize("gam1", [0.0, 1e-9, -0.2, 8.0 / 15.0])
def test_steps(mhd3d, oracle, gam1, lmag, lrot):
    _gpu_or_skip(mhd3d)
    su = mhd3d.make_setup(_cfg(mhd3d, 40, 9, 13, lmag=lmag, lrot=lrot))
    su.params.gam1 = gam1
    st = _random_state(mhd3d, su, amp=0.01)
    o = oracle.Oracle(su.params, su.grid, st)
    g = mhd3d.GpuSim(su, mode=mhd3d.MODE_FAST)
    g.upload(st)
    ro, rg = o.step(3), g.step(3)
    assert ro["status"] == 0 and rg["nit"] == 3
    got, ref = g.download(), o.get_state()
    g.close()
    for f in _fields(su.params):
        a, b = got[f][1:-1, 1:-1, 1:-1], ref[f][1:-1, 1:-1, 1:-1]
        assert np.abs(a - b).max() <= FAST_TOL * np.abs(b).max(), f
