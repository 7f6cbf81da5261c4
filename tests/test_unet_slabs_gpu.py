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


@pytest.mark.parametrize("h,w,n", [(8, 16, 96), (8, 64, 64), (8, 32, 61)])
def test_several_tiles_per_block_on_narrow_rows(h, w, n):
    """batches at which a block takes two or four tiles of the line of pixels: the outputs, exactly"""
    torch = pytest.importorskip("torch")
    from lbm_mirror_gb300 import UNet
    from tests.test_unet_gradient_passes_gpu import _oracle, _whole_params
    widths = (48, 16, 32, 16)
    gen = torch.Generator().manual_seed(19)
    net = UNet(height=h, width=w, widths=widths, out_channels=2, max_batch=n, seed=3)
    params = _whole_params(gen, widths, 2)
    net.set_params(params.numpy())
    x = torch.randint(-2, 3, (n, h, w, 16), generator=gen).float()
    y, _ = _oracle(params, x, torch.zeros((n, h, w, 2)), widths, 2)
    xin = x.to(torch.bfloat16).cuda()
    out = torch.empty((n, h, w, 2), device="cuda")
    torch.cuda.synchronize()
    net.set_input(xin.data_ptr(), n)
    net.forward(n, out.data_ptr())
    net.synchronize()
    assert (out.cpu().numpy() == y).all()
