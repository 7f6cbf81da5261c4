"""Channel counts that the convolutions hold in slabs of 64, 32 and 16 channels, in each form: rows of
128 pixels and more (resident weights and halo), rows of 64 to 16 (three shifted halos), an output split
over two blocks.  Exact inputs and the bound of test_unet_gradient_passes_gpu (at most 2,880 pixels)."""
import pytest

from tests.test_unet_gradient_passes_gpu import test_gradients_at_the_edges_of_the_split as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,n,widths", [
    (16, 128, 1, (64, 48, 32, 16)),
    (8, 256, 1, (32, 96, 128, 64)),
    (16, 128, 1, (48, 96, 128, 128)),
    (16, 128, 1, (128, 64, 48, 192)),
    (32, 64, 1, (64, 128, 96, 48)),
    (8, 128, 2, (16, 32, 64, 128)),
])
def test_slabs(h, w, n, widths):
    check(h, w, n, widths, 3, 0)
