"""Steps captured in a CUDA graph on the caller's stream: a replay takes the
steps that a call would.  A call that starts from a synced state clears an
earlier stop, and so does a replay, when the stop came after the capture as well."""
import numpy as np
import pytest

from test_gpu_parity import _gpu_or_skip

pytestmark = pytest.mark.gpu

MHD3D_ERR_TIMEOUT = 6


@pytest.mark.parametrize("mode,stopped", [("EXACT", False), ("FAST", False), ("FP32", False),
                                          ("EXACT", True), ("FAST", True)])
def test_replay(mhd3d, mode, stopped):
    _gpu_or_skip(mhd3d)
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda")
    su = mhd3d.make_setup(mhd3d.convection_config(40, 24, 36, ra=1e6, ta=1e6))
    a, b = (mhd3d.GpuSim(su, mode=getattr(mhd3d, "MODE_" + mode)) for _ in range(2))
    for g in (a, b):
        g.upload(su.state)
        g.step(2)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    a.set_stream(stream.cuda_stream)
    with torch.cuda.graph(graph, stream=stream):
        a.step_async(4)
    assert a.sync()["nit"] == 2   # nothing has run yet
    if stopped:   # a step that gives up at once, before it writes anything
        a.set_wait_limit(0)
        r = a.step(1, check=False)
        assert r["status"] == MHD3D_ERR_TIMEOUT and r["nit"] == 2
        a.set_wait_limit(1 << 22)
    with torch.cuda.stream(stream):
        graph.replay()
    ra, rb = a.sync(check=False), b.step(4)
    assert ra == rb and ra["nit"] == 6
    da, db = a.download(), b.download()
    for f in mhd3d.FIELDS:
        assert np.array_equal(da[f], db[f]), f
    a.set_stream(None)
    del graph
    a.close()
    b.close()
