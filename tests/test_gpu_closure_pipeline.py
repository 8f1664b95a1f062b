"""The convolution kernels on grids that give every CTA several tiles: the
input ring and the stages of the weight gradient are reused, their barriers
wrap, full and short segments follow each other in one stage, and sums run
over several segments.  Bounds and checker as in test_gpu_closure.py."""
import pytest

from test_gpu_closure import test_conv3d_forward_and_gradients as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("shape", [(16, 40, 70), (12, 40, 130), (40, 37, 13), (9, 50, 128)])
def test_many_tiles_a_cta(mhd3d, shape, cin, cout):
    _check(mhd3d, shape, cin, cout)
