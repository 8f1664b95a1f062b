"""The convolutions at x periods around the tiles of the forward pass (128
voxels) and of the weight gradient (64), and the smallest: the last segment's
own boxes, halos and K steps."""
import pytest

from test_gpu_closure import test_conv3d_forward_and_gradients as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("nx", [1, 2, 13, 14, 15, 62, 63, 65, 127, 129, 130, 191])
def test_tails(mhd3d, nx, cin, cout):
    _check(mhd3d, (3, 4, nx), cin, cout)
