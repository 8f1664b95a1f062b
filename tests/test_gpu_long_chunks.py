"""The FP64 stage kernels where a chunk of z planes is long, as on large grids:
the plane ring and the Z slots are reused many times.  192x148 cells are 222
tiles, so the rule takes chunks of 37 planes (one wave, at most 40 planes a
chunk).  Bounds as in test_gpu_parity.py."""
import numpy as np
import pytest

from test_gpu_parity import FAST_TOL, _cfg, _fields, _gpu_or_skip, _random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["EXACT", "FAST"])
@pytest.mark.parametrize("lmag", [1, 0])
def test_long_chunks(mhd3d, oracle, lmag, mode):
    _gpu_or_skip(mhd3d)
    su = mhd3d.make_setup(_cfg(mhd3d, 192, 148, 74, lmag=lmag))
    st = _random_state(mhd3d, su, amp=0.01)
    o = oracle.Oracle(su.params, su.grid, st)
    g = mhd3d.GpuSim(su, mode=getattr(mhd3d, "MODE_" + mode))
    g.upload(st)
    o.step(2)
    g.step(2)
    got, ref = g.download(), o.get_state()
    g.close()
    for f in _fields(su.params):
        a, b = got[f][1:-1, 1:-1, 1:-1], ref[f][1:-1, 1:-1, 1:-1]
        if mode == "EXACT":
            assert np.array_equal(a, b), f
        else:
            assert np.abs(a - b).max() <= FAST_TOL * np.abs(b).max(), f
