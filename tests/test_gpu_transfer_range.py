"""A device array that ends before its field does is refused, as the copy of it
always was, and not read or written past its end.  The bytes behind the short
array belong to the next allocation of this process, so nothing unmapped is
named even where no check is made."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import _cfg, _gpu_or_skip

pytestmark = pytest.mark.gpu

MHD3D_ERR_CUDA = 2


def _neighbours(rt, size, want):
    """Allocations of `size` bytes, one of them followed at once by others that reach `want` bytes."""
    ptrs = []
    for _ in range(64):
        p = C.c_void_p()
        assert rt.cudaMalloc(C.byref(p), C.c_size_t(size)) == 0
        ptrs.append(p.value)
    have = set(ptrs)
    for p in ptrs:
        if all(p + i * size in have for i in range(1, -(-want // size))):
            return p, ptrs
    return None, ptrs


@pytest.mark.parametrize("way", ["upload", "download"])
def test_short_device_array(mhd3d, way):
    _gpu_or_skip(mhd3d)
    torch = pytest.importorskip("torch")
    rt = C.CDLL("libcudart.so.12")
    su = mhd3d.make_setup(_cfg(mhd3d, 14, 14, 14, lmag=0))
    n = int(np.prod(su.shape))
    g = mhd3d.GpuSim(su, mode=mhd3d.MODE_EXACT)
    g.upload(su.state)
    dev = [torch.from_numpy(np.ascontiguousarray(su.state[f].ravel(order="F"))).cuda() for f in mhd3d.FIELDS[:5]]
    torch.cuda.synchronize()
    size = 16384   # half of a field
    short, ptrs = _neighbours(rt, size, 8 * n)
    try:
        if short is None:
            pytest.skip("no adjacent allocations")
        args = [C.c_void_p(t.data_ptr()) for t in dev]
        args[2] = C.c_void_p(short)
        call = g.lib.mhd3d_upload if way == "upload" else g.lib.mhd3d_download
        assert call(g.h, *args, None, None, None) == MHD3D_ERR_CUDA
        g.upload(su.state)   # the handle is usable
        assert g.step(1)["nit"] == 1
    finally:
        g.close()
        for p in ptrs:
            rt.cudaFree(C.c_void_p(p))
