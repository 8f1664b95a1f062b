"""Horizontal means at planes that one CTA holds, that CTAs share unevenly,
and with more planes than the device holds CTAs at once, with and without a
magnetic field, against the oracle (bounds as in test_gpu_profiles.py)."""
import numpy as np
import pytest

from test_gpu_parity import _cfg, _gpu_or_skip, _random_state
from test_gpu_profiles import PROF_FP32, PROF_FP64, _rel, _rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmag", [True, False])
@pytest.mark.parametrize("nx,ny,nz", [(4, 4, 4), (33, 9, 6), (31, 67, 5), (12, 8, 603)])
def test_profile_split(mhd3d, oracle, nx, ny, nz, lmag):
    _gpu_or_skip(mhd3d)
    su = mhd3d.make_setup(_cfg(mhd3d, nx, ny, nz, lmag=lmag))
    st = _random_state(mhd3d, su, amp=0.05)
    ref = oracle.Oracle(su.params, su.grid, st).profiles()
    for mode, tol in ((mhd3d.MODE_FAST, PROF_FP64), (mhd3d.MODE_FP32, PROF_FP32)):
        g = mhd3d.GpuSim(su, mode=mode)
        g.upload(st)
        r = _rel(g.profiles(), ref)
        assert np.all(r[_rows(mhd3d, su.params)] <= tol), (mode, r)
        g.close()
