"""Upload and download of device arrays in place against the host arrays' path:
ragged rows around the kernels' strides, partial field lists, arrays that are
misaligned or overlap (which go through the staging fields), both buffers."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import _cfg, _fields, _gpu_or_skip, _random_state

pytestmark = pytest.mark.gpu


def _p(t, off=0):
    return None if t is None else C.c_void_p(t.data_ptr() + off)


@pytest.mark.parametrize("mode", ["MODE_EXACT", "MODE_FP32"])
@pytest.mark.parametrize("size", [(2, 2, 4), (30, 6, 5), (31, 7, 5), (126, 9, 4), (127, 5, 6), (300, 3, 7)])
def test_device_arrays_equal_host_arrays(mhd3d, size, mode):
    _gpu_or_skip(mhd3d)
    torch = pytest.importorskip("torch")
    su = mhd3d.make_setup(_cfg(mhd3d, *size))
    st = _random_state(mhd3d, su, seed=size[0])
    f = _fields(su.params)
    n = int(np.prod(su.shape))
    a, b = (mhd3d.GpuSim(su, mode=getattr(mhd3d, mode)) for _ in range(2))
    dev = [torch.from_numpy(np.ascontiguousarray(st[k].ravel(order="F"))).cuda() for k in f]
    odd = torch.empty(8 * n + 4, dtype=torch.uint8, device="cuda")   # a field on 4 bytes
    odd[4:] = dev[3].view(torch.uint8)
    torch.cuda.synchronize()
    for steps in (0, 1):   # the second time the other buffer is the current one
        for ptrs in ([_p(t) for t in dev], [_p(t) for t in dev[:3]] + [_p(odd, 4)] + [_p(t) for t in dev[4:]]):
            a.upload(st)
            assert b.lib.mhd3d_upload(b.h, *ptrs) == 0
            a.step(1 + steps)
            b.step(1 + steps)
            ref = a.download()
            out = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in f]
            torch.cuda.synchronize()
            assert b.lib.mhd3d_download(b.h, *[_p(t) for t in out]) == 0
            for k, t in zip(f, out):
                assert np.array_equal(t.cpu().numpy(), ref[k].ravel(order="F")), k
            # some fields only; the last of two arrays in one place wins
            out[1].zero_()
            torch.cuda.synchronize()
            assert b.lib.mhd3d_download(b.h, *[_p(out[1]), _p(out[1])] + [None] * 6) == 0
            assert np.array_equal(out[1].cpu().numpy(), ref[f[1]].ravel(order="F"))
    a.close()
    b.close()
