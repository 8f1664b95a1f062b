"""The weight gradient in a caller's workspace: the same bits as in the
allocator's, whatever the workspace held, for grids below and above one
segment per SM; a workspace that is too small is refused."""
import ctypes as C

import pytest

from test_gpu_parity import _gpu_or_skip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 70), (7, 9, 130)])
def test_workspace(mhd3d, shape, cin, cout):
    _gpu_or_skip(mhd3d)
    torch = pytest.importorskip("torch")
    lib = mhd3d.gpu_lib()
    nz, ny, nx = shape
    g = torch.Generator().manual_seed(cin + cout)
    x = torch.randn(shape + (cin,), generator=g).to(torch.bfloat16).cuda()
    dy = torch.randn(shape + (cout,), generator=g).to(torch.bfloat16).cuda()
    p = lambda t: C.c_void_p(t.data_ptr())
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    size = lib.mhd3d_conv3d_wgrad_workspace(cin, cout)
    ws = torch.full((size,), 255, dtype=torch.uint8, device="cuda")   # NaN partials, a set error flag
    out = []
    for own in (True, False):
        dw = torch.zeros((cout, 27 * cin), dtype=torch.float32, device="cuda")
        db = torch.zeros(cout, dtype=torch.float32, device="cuda")
        if own:
            assert lib.mhd3d_conv3d_wgrad(cin, cout, p(x), p(dy), p(dw), p(db), nx, ny, nz, s) == 0
        else:
            assert lib.mhd3d_conv3d_wgrad_ws(cin, cout, p(x), p(dy), p(dw), p(db), nx, ny, nz, p(ws), size, s) == 0
        out.append((dw, db))
    assert all(torch.equal(a, b) for a, b in zip(*out))
    assert bool(torch.isfinite(out[1][0]).all())
    grid = min(torch.cuda.get_device_properties(0).multi_processor_count, (nx + 63) // 64 * ny * nz)
    need = grid * (cout * 27 * cin + cout) * 4 + 16
    assert lib.mhd3d_conv3d_wgrad_ws(cin, cout, p(x), p(dy), p(dw), p(db), nx, ny, nz, p(ws), need - 1, s) == 1
    assert lib.mhd3d_conv3d_wgrad_workspace(16, 16) == -1
