"""The 12 subgrid targets of the box filter in both storage types, with and
without a magnetic field, by 4 (its own kernel) and by other factors, against
numpy on the downloaded state.  A target is a difference of two filtered
products, rounded to FP32 at the end: at most 64 FP64 terms each, so 128 eps64
of the larger product and one FP32 rounding."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import _cfg, _gpu_or_skip, _random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["FAST", "FP32"])
@pytest.mark.parametrize("lmag", [1, 0])
@pytest.mark.parametrize("fac", [2, 3, 4, 6])
def test_targets(mhd3d, fac, lmag, mode):
    _gpu_or_skip(mhd3d)
    torch = pytest.importorskip("torch")
    n = (36, 12, 24)
    su = mhd3d.make_setup(_cfg(mhd3d, *n, lmag=lmag))
    g = mhd3d.GpuSim(su, mode=getattr(mhd3d, "MODE_" + mode))
    g.upload(_random_state(mhd3d, su, amp=0.05))
    st = g.download()
    m = [v // fac for v in n]
    cs = torch.zeros((8 if lmag else 5) * int(np.prod([v + 2 for v in m])), dtype=torch.float64, device="cuda")
    tg = torch.zeros((m[2], m[1], m[0], 12), dtype=torch.float32, device="cuda")
    assert g.lib.mhd3d_coarsen(g.h, fac, C.c_void_p(cs.data_ptr()), C.c_void_p(tg.data_ptr()), None) == 0
    torch.cuda.synchronize()
    g.close()

    def box(a):
        return a.reshape(m[0], fac, m[1], fac, m[2], fac).mean(axis=(1, 3, 5))

    x = {f: st[f][1:-1, 1:-1, 1:-1] for f in mhd3d.FIELDS if st[f] is not None}
    ro, mom = x["ro"], [x["ru"], x["rv"], x["rw"]]
    u = [a / ro for a in mom]
    R, M, E = box(ro), [box(a) for a in mom], box(ro * x["tt"])
    V = [a / R for a in M]
    pairs = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
    terms = [(box(mom[a] * u[b]), M[a] * V[b]) for a, b in pairs]
    terms += [(box(mom[a] * x["tt"]), M[a] * E / R) for a in range(3)]
    if lmag:
        b = [x["bx"], x["by"], x["bz"]]
        B = [box(a) for a in b]
        for i, j in ((1, 2), (2, 0), (0, 1)):
            terms.append((box(u[i] * b[j] - u[j] * b[i]), V[i] * B[j] - V[j] * B[i]))
    else:
        terms += [(np.zeros(m), np.zeros(m))] * 3
    got = tg.double().cpu().numpy()
    for c, (p, q) in enumerate(terms):
        ref = np.transpose(p - q, (2, 1, 0))
        size = max(np.abs(p).max(), np.abs(q).max())
        if c >= 9 and lmag:   # the products whose difference each side already is
            i, j = ((1, 2), (2, 0), (0, 1))[c - 9]
            size = max(size, *(np.abs(u[s]).max() * np.abs(b[t]).max() for s, t in ((i, j), (j, i))))
        assert np.abs(got[..., c] - ref).max() <= 2.0 ** -24 * np.abs(ref).max() + 128 * 2.0 ** -52 * size, c
