"""Adam on several tensors in one call: the bits of one call a tensor, at
sizes from one value to several grid strides and more tensors than a launch takes."""
import ctypes as C

import pytest

from test_gpu_parity import _gpu_or_skip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1], [27648, 32, 13824, 16], [5, 300001] + [7 + i for i in range(17)]])
def test_adam_multi(mhd3d, sizes):
    _gpu_or_skip(mhd3d)
    torch = pytest.importorskip("torch")
    import closure
    lib = mhd3d.gpu_lib()
    gen = torch.Generator().manual_seed(len(sizes))
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def rand(n):
        return torch.randn(n, generator=gen).cuda()

    one = [[rand(n), rand(n), 0.1 * rand(n), rand(n).square(), torch.zeros(n, dtype=torch.bfloat16, device="cuda")]
           for n in sizes]
    many = [[t.clone() for t in r] for r in one]
    args = (1e-3, 0.9, 0.999, 1e-8, 3)
    for i, (p, g, m, v, c) in enumerate(one):
        assert lib.mhd3d_adam(*[C.c_void_p(t.data_ptr()) for t in (p, g, m, v)], p.numel(), *args,
                              C.c_void_p(c.data_ptr()) if i % 2 else None, s) == 0
    tab = (closure._AdamTensor * len(many))(*[
        (p.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(), p.numel(), c.data_ptr() if i % 2 else None)
        for i, (p, g, m, v, c) in enumerate(many)])
    assert lib.mhd3d_adam_multi(tab, len(many), *args, s) == 0
    torch.cuda.synchronize()
    for a, b in zip(one, many):
        assert all(torch.equal(x, y) for x, y in zip(a, b))
    tab[len(many) - 1].n = 0
    before = many[0][0].clone()
    assert lib.mhd3d_adam_multi(tab, len(many), *args, s) == 1
    torch.cuda.synchronize()
    assert torch.equal(before, many[0][0])
