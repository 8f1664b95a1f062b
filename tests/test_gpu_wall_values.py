"""Wall values that BCON leaves to the right-hand side: BZ on both walls when
IBC is not 0 (3dmhdsub.f:2871-2878, 2947-2954 rewrite it for IBC=0 only), TT on
the top wall when ITC is 3 (2833-2868 rewrite it for the others).  They take
the RK3 update like any cell, Z included, so every mode is held to its bounds
against the oracle on the walls too."""
import numpy as np
import pytest

from test_gpu_fp32 import STEP_FULL
from test_gpu_parity import FAST_TOL, _cfg, _fields, _gpu_or_skip, _random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["EXACT", "FAST", "FP32"])
@pytest.mark.parametrize("kw", [dict(ibcon=1), dict(ibcon=1, lrot=0, izcon=0, itcon=1), dict(itcon=3),
                                dict(itcon=3, lmag=0), dict(itcon=3, ibcon=1)])
def test_wall_values_take_the_update(mhd3d, oracle, kw, mode):
    _gpu_or_skip(mhd3d)
    su = mhd3d.make_setup(_cfg(mhd3d, 36, 10, 13, **kw))
    st = _random_state(mhd3d, su, amp=0.01)
    o = oracle.Oracle(su.params, su.grid, st)
    g = mhd3d.GpuSim(su, mode=getattr(mhd3d, "MODE_" + mode))
    g.upload(st)
    o.step(3)
    g.step(3)
    got, ref = g.download(), o.get_state()
    g.close()
    for f in _fields(su.params):
        a, b = got[f][1:-1, 1:-1, 1:-1], ref[f][1:-1, 1:-1, 1:-1]
        if mode == "EXACT":
            assert np.array_equal(a, b), (f, np.abs(a - b).max())
        else:
            err = np.abs(a - b).max() / np.abs(b).max()
            assert err <= (FAST_TOL if mode == "FAST" else STEP_FULL), (f, err)
