"""The column-march stage kernels at the sizes where their bookkeeping can go
wrong: the smallest grids, one-plane remainders of z chunks, ragged tiles and
rows of one cell more than a tile, with live walls and ghost planes, against
the CPU oracle.  The tolerance is that of the FMA mode's parity test."""
import numpy as np
import pytest

from test_gpu_parity import FAST_TOL, _cfg, _fields, _gpu_or_skip, _random_state

pytestmark = pytest.mark.gpu

SIZES = [(2, 2, 4), (3, 2, 5), (32, 4, 8), (33, 5, 9), (31, 3, 13), (65, 9, 131), (96, 7, 12)]


@pytest.mark.parametrize("mag,rot", [(1, 1), (0, 0)])
@pytest.mark.parametrize("size", SIZES)
def test_fast_steps_at_edges(mhd3d, oracle, size, mag, rot):
    _gpu_or_skip(mhd3d)
    su = mhd3d.make_setup(_cfg(mhd3d, *size, lmag=mag, lrot=rot))
    st = _random_state(mhd3d, su, seed=sum(size))
    orc = oracle.Oracle(su.params, su.grid, st)
    orc.step(3)
    ref = orc.get_state()
    g = mhd3d.GpuSim(su, mode=mhd3d.MODE_FAST)
    g.upload(st)
    g.step(3)
    got = g.download()
    g.close()
    for f in _fields(su.params):
        a, b = got[f][1:-1, 1:-1, 1:-1], ref[f][1:-1, 1:-1, 1:-1]
        assert np.abs(a - b).max() <= FAST_TOL * max(np.abs(b).max(), 1e-300), f
