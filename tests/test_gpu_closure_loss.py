"""The closure loss and its gradient where the arrays allow 16-byte accesses and
where they do not (offset by one element), for voxel counts around a block."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import _gpu_or_skip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("nvox", [1, 63, 64, 65, 4097])
def test_loss_and_gradient(mhd3d, nvox, off):
    _gpu_or_skip(mhd3d)
    torch = pytest.importorskip("torch")
    lib = mhd3d.gpu_lib()
    rng = np.random.default_rng(nvox + off)
    p, t = (rng.standard_normal((nvox, n)).astype(np.float32) for n in (16, 12))
    dp = torch.zeros(nvox * 16 + off, dtype=torch.float32, device="cuda")
    dt = torch.zeros(nvox * 12 + off, dtype=torch.float32, device="cuda")
    dp[off:], dt[off:] = torch.from_numpy(p.ravel()).cuda(), torch.from_numpy(t.ravel()).cuda()
    dy = torch.ones(nvox * 16 + off, dtype=torch.bfloat16, device="cuda")
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert lib.mhd3d_closure_loss(C.c_void_p(dp.data_ptr() + 4 * off), C.c_void_p(dt.data_ptr() + 4 * off), nvox,
                                  C.c_void_p(dy.data_ptr() + 2 * off), C.c_void_p(loss.data_ptr()), C.c_void_p(s)) == 0
    d = p[:, :12].astype(np.float64) - t
    g = np.zeros((nvox, 16))
    g[:, :12] = 2 * d / (12 * nvox)
    assert abs(loss.item() - (d * d).sum() / (12 * nvox)) <= 1e-12 * (d * d).sum() / (12 * nvox)
    got = dy[off:].float().cpu().numpy().reshape(nvox, 16)
    ref = torch.from_numpy(g).float().to(torch.bfloat16).float().numpy()   # FP32, then BF16, as the gradient is stored
    assert np.array_equal(got, ref)
