"""The convective flux of planes with a temperature outlier, in any corner:
its deviations may be taken from any value near the plane's mean, but not from
the outlier.  Against extended precision on the uploaded state: 64 roundings
of the terms and of the mean temperature."""
import numpy as np
import pytest

from test_gpu_parity import _cfg, _gpu_or_skip, _random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", [(1, 1), (-2, -2), (1, -2), (40, 33)])
@pytest.mark.parametrize("n", [(128, 96, 8), (67, 45, 6)])
def test_fconv_beside_an_outlier(mhd3d, n, where):
    _gpu_or_skip(mhd3d)
    su = mhd3d.make_setup(_cfg(mhd3d, *n))
    st = _random_state(mhd3d, su)
    st["tt"][where[0], where[1], :] *= 1e4
    mhd3d.wrap_periodic(st["tt"])
    g = mhd3d.GpuSim(su, mode=mhd3d.MODE_FAST)
    g.upload(st)
    got = g.profiles()[mhd3d.PROFILES.index("fconv")]
    g.close()
    x = {f: st[f][1:-1, 1:-1, 1:-1].astype(np.longdouble) for f in mhd3d.FIELDS[:5]}
    mean = lambda a: a.mean(axis=(0, 1))
    ttm = mean(x["tt"])
    ke = sum((x[f] / x["ro"]) ** 2 for f in ("ru", "rv", "rw"))
    ref = mean(-x["rw"] * (np.longdouble(2.5) * (x["tt"] - ttm) + ke / 2))
    size = mean(np.abs(x["rw"]) * (2.5 * np.abs(x["tt"] - ttm) + ke / 2)) + 2.5 * np.abs(ttm) * mean(np.abs(x["rw"]))
    err = np.abs(got - ref)
    assert np.all(err <= 64 * 2.0 ** -52 * size), np.max(err / size) / 2.0 ** -52
