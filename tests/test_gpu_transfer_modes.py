"""Device arrays in place against host arrays in the FMA build, the one that
reads what its output buffer held before the step, and several launches in a
row on the caller's stream: the same bits whichever way the state came in."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import _cfg, _fields, _gpu_or_skip, _random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(2, 2, 4), (31, 7, 5), (127, 5, 6), (96, 9, 20)])
@pytest.mark.parametrize("lmag", [1, 0])
def test_fma_build(mhd3d, size, lmag):
    _gpu_or_skip(mhd3d)
    torch = pytest.importorskip("torch")
    su = mhd3d.make_setup(_cfg(mhd3d, *size, lmag=lmag))
    st = _random_state(mhd3d, su, seed=size[0], amp=0.01)
    f = _fields(su.params)
    n = int(np.prod(su.shape))
    a, b = (mhd3d.GpuSim(su, mode=mhd3d.MODE_FAST) for _ in range(2))
    stream = torch.cuda.Stream()
    dev = [torch.from_numpy(np.ascontiguousarray(st[k].ravel(order="F"))).cuda() for k in f]
    none = [None] * (8 - len(f))
    torch.cuda.synchronize()
    b.set_stream(stream.cuda_stream)
    for steps in (1, 2, 3):   # from either buffer
        a.upload(st)
        assert b.lib.mhd3d_upload(b.h, *[C.c_void_p(t.data_ptr()) for t in dev], *none) == 0
        ra = a.step(steps)
        for _ in range(steps):
            b.step_async(1)
        assert b.sync() == ra
        out = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in f]
        torch.cuda.synchronize()
        assert b.lib.mhd3d_download(b.h, *[C.c_void_p(t.data_ptr()) for t in out], *none) == 0
        ref = a.download()
        for k, t in zip(f, out):
            assert np.array_equal(t.cpu().numpy(), ref[k].ravel(order="F")), k
    b.set_stream(None)
    a.close()
    b.close()
