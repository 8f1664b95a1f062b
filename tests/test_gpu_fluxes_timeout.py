"""A right-hand side whose bounded wait gives up says so and leaves the run
alone: the next step advances as if it had not been asked for."""
import numpy as np
import pytest

from test_gpu_parity import _gpu_or_skip

pytestmark = pytest.mark.gpu

MHD3D_ERR_TIMEOUT = 6


@pytest.mark.parametrize("mode", ["EXACT", "FAST"])
def test_fluxes_report_their_timeout_and_the_run_goes_on(mhd3d, mode):
    _gpu_or_skip(mhd3d)
    su = mhd3d.make_setup(mhd3d.convection_config(40, 24, 36, ra=1e6, ta=1e6))
    a, b = (mhd3d.GpuSim(su, mode=getattr(mhd3d, "MODE_" + mode)) for _ in range(2))
    for g in (a, b):
        g.upload(su.state)
        g.step(1)
    a.set_wait_limit(0)
    with pytest.raises(mhd3d.Mhd3dError) as e:
        a.fluxes()
    assert e.value.code == MHD3D_ERR_TIMEOUT
    a.set_wait_limit(1 << 22)
    assert a.sync()["status"] == 0
    ra, rb = a.step(2, check=False), b.step(2)
    assert ra == rb and ra["nit"] == 3
    fa, fb = a.fluxes(), b.fluxes()
    sa, sb = a.download(), b.download()
    for x, y in [(fa[k], fb[k]) for k in fa] + [(sa[k], sb[k]) for k in mhd3d.FIELDS]:
        assert np.array_equal(x, y)
    a.close()
    b.close()
