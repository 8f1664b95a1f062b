"""The box filter by 4 (its own kernel) and by other factors against numpy
means of the downloaded state, in both storage types, with and without a
magnetic field.  Sums of at most 64 positive or mixed FP64 terms: 64 eps of
the largest term."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import _cfg, _gpu_or_skip, _random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["FAST", "FP32"])
@pytest.mark.parametrize("lmag", [1, 0])
@pytest.mark.parametrize("fac", [2, 3, 4])
def test_coarsen(mhd3d, fac, lmag, mode):
    _gpu_or_skip(mhd3d)
    torch = pytest.importorskip("torch")
    n = (36, 12, 24)
    su = mhd3d.make_setup(_cfg(mhd3d, *n, lmag=lmag))
    g = mhd3d.GpuSim(su, mode=getattr(mhd3d, "MODE_" + mode))
    g.upload(_random_state(mhd3d, su, amp=0.05))
    st = g.download()
    m = [v // fac for v in n]
    nf = 8 if lmag else 5
    full = tuple(v + 2 for v in m)
    cs = torch.zeros(nf * int(np.prod(full)), dtype=torch.float64, device="cuda")
    tg = torch.empty(int(np.prod(m)) * 12, dtype=torch.float32, device="cuda")
    assert g.lib.mhd3d_coarsen(g.h, fac, C.c_void_p(cs.data_ptr()), C.c_void_p(tg.data_ptr()), None) == 0
    torch.cuda.synchronize()
    g.close()
    got = {f: a.reshape(full, order="F")[1:-1, 1:-1, 1:-1]
           for f, a in zip(mhd3d.FIELDS, cs.cpu().numpy().reshape(nf, -1))}

    def mean(a):
        return a.reshape(m[0], fac, m[1], fac, m[2], fac).mean(axis=(1, 3, 5))

    x = {f: st[f][1:-1, 1:-1, 1:-1] for f in mhd3d.FIELDS[:nf]}
    for f in mhd3d.FIELDS[:nf]:
        ref = mean(x["ro"] * x["tt"]) / mean(x["ro"]) if f == "tt" else mean(x[f])
        assert np.abs(got[f] - ref).max() <= 64 * 2.0 ** -52 * np.abs(x[f]).max(), f
    assert np.isfinite(tg.cpu().numpy()).all()
