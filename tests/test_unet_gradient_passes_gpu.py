"""The passes that form a layer's output gradient (ReLU, upsample or pool
gradient and bias sums in one pass; the head's backward pass) at the edges of
their work split: one to eight outputs, channel counts that do not divide the
block (48, 80), more than 256 channels (bias sums in a pass of their own),
fewer pixels than blocks.

Weights of -1, 0 and 1 (two taps per output channel), small whole inputs and a
target that makes the output's gradient a few eighths keep every sum of a
convolution exact in FP32, so the network and an FP64 restatement that rounds
to bf16 where the network rounds hold the same activations and gradients.  What
is left is the FP32 sums of the weight and bias gradients over at most M =
2,880 pixels: M x 2^-24 < 2^-12 of the sum of magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

BOUND = 2.0 ** -12


class _Round(torch.autograd.Function):
    """bf16 rounding of the value and of its gradient"""

    @staticmethod
    def forward(ctx, x):
        return x.to(torch.bfloat16).to(x.dtype)

    @staticmethod
    def backward(ctx, g):
        return g.to(torch.bfloat16).to(g.dtype)


class _RoundGrad(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x

    @staticmethod
    def backward(ctx, g):
        return g.to(torch.bfloat16).to(g.dtype)


def _oracle(params, x, dy, widths, outs):
    """output and parameter gradients for the output gradient dy; NHWC, weights (co, ky, kx, ci), bias after each"""
    f = torch.nn.functional
    w = widths
    layers = [(w[0], 16), (w[0], w[0]), (w[1], w[0]), (w[1], w[1]), (w[2], w[1]), (w[2], w[2]), (w[3], w[2]),
              (w[3], w[3]), (w[2], w[3] + w[2]), (w[2], w[2]), (w[1], w[2] + w[1]), (w[1], w[1]),
              (w[0], w[1] + w[0]), (w[0], w[0])]
    leaves, o = [], 0
    for co, ci in layers:
        n = co * 9 * ci
        k = params[o:o + n].to(torch.bfloat16).double().reshape(co, 3, 3, ci).requires_grad_()
        b = params[o + n:o + n + co].double().requires_grad_()
        leaves += [k, b]
        o += n + co
    hw = params[o:o + outs * w[0]].double().reshape(outs, w[0]).requires_grad_()
    hb = params[o + outs * w[0]:].double().requires_grad_()
    leaves += [hw, hb]

    def conv(li, a):
        z = f.conv2d(a, leaves[2 * li].permute(0, 3, 1, 2), leaves[2 * li + 1], padding=1)
        return _Round.apply(torch.relu(_RoundGrad.apply(z)))

    def up(a):
        return _RoundGrad.apply(a).repeat_interleave(2, 2).repeat_interleave(2, 3)

    a = x.double().permute(0, 3, 1, 2)
    skips = []
    for lvl in range(3):
        a = conv(2 * lvl + 1, conv(2 * lvl, a))
        skips.append(a)
        a = _Round.apply(f.avg_pool2d(a, 2))
    a = conv(7, conv(6, a))
    for k, lvl in enumerate((2, 1, 0)):
        a = conv(9 + 2 * k, conv(8 + 2 * k, _RoundGrad.apply(torch.cat([up(a), skips[lvl]], 1))))
    y = torch.einsum("nchw,oc->nhwo", _RoundGrad.apply(a), hw) + hb
    y.backward(dy.double())
    return y.detach().numpy(), [p.grad.reshape(-1).numpy() for p in leaves]


def _whole_params(gen, widths, outs):
    """two taps of -1 or 1 per output channel (conv layers), biases 0 or 1, head weights -1, 0 or 1"""
    w = widths
    out = []
    for co, ci in [(w[0], 16), (w[0], w[0]), (w[1], w[0]), (w[1], w[1]), (w[2], w[1]), (w[2], w[2]), (w[3], w[2]),
                   (w[3], w[3]), (w[2], w[3] + w[2]), (w[2], w[2]), (w[1], w[2] + w[1]), (w[1], w[1]),
                   (w[0], w[1] + w[0]), (w[0], w[0])]:
        k = torch.zeros((co, 9 * ci))
        at = torch.randint(0, 9 * ci, (co, 2), generator=gen)
        k.scatter_(1, at, torch.randint(0, 2, (co, 2), generator=gen) * 2.0 - 1.0)
        out += [k.reshape(-1), torch.randint(0, 2, (co,), generator=gen).float()]
    out += [torch.randint(-1, 2, (outs * w[0],), generator=gen).float(), torch.zeros(outs)]
    return torch.cat(out)


CASES = [
    # h, w, batch, widths, outputs, conv kernel (0 tcgen05, 1 mma.sync)
    pytest.param(8, 16, 1, (16, 16, 32, 16), 1, 0, id="1out_tiny"),
    pytest.param(24, 40, 3, (48, 80, 16, 32), 2, 0, id="2out_48_80"),
    pytest.param(16, 16, 2, (80, 48, 32, 48), 5, 1, id="5out_80_48"),
    pytest.param(16, 16, 1, (272, 16, 16, 16), 3, 1, id="3out_272"),
    pytest.param(8, 16, 2, (32, 16, 288, 16), 8, 1, id="8out_288"),
]


@pytest.mark.parametrize("h,w,n,widths,outs,kind", CASES)
def test_gradients_at_the_edges_of_the_split(h, w, n, widths, outs, kind):
    from lbm_mirror_gb300 import UNet
    gen = torch.Generator().manual_seed(11)
    net = UNet(height=h, width=w, widths=widths, out_channels=outs, max_batch=n, seed=3)
    net.set_conv_kernel(kind)
    params = _whole_params(gen, widths, outs)
    net.set_params(params.numpy())
    x = torch.randint(-2, 3, (n, h, w, 16), generator=gen).float()
    dy = torch.randint(-4, 5, (n, h, w, outs), generator=gen).float() / 8
    y, grads = _oracle(params, x, dy, widths, outs)
    # 2 (y - t) / size = dy
    tgt = torch.from_numpy(y) - dy.double() * dy.numel() / 2
    assert torch.equal(tgt.float().double(), tgt)
    xin, tg = x.to(torch.bfloat16).cuda(), tgt.float().cuda()
    out = torch.empty((n, h, w, outs), device="cuda")
    torch.cuda.synchronize()
    net.set_input(xin.data_ptr(), n)
    net.forward(n, out.data_ptr())
    net.backward(tg.data_ptr(), n)
    net.synchronize()
    got = net.grads().astype(np.float64)
    assert np.array_equal(out.cpu().numpy(), y)
    o = 0
    for k, b in enumerate(grads):
        a = got[o:o + b.size]
        o += b.size
        assert np.linalg.norm(a - b) <= BOUND * np.linalg.norm(b), (k, np.linalg.norm(a - b) / np.linalg.norm(b))
    assert o == got.size


@pytest.mark.parametrize("own_stream", [True, False], ids=["net_stream", "caller_stream"])
def test_gradients_repeat_bit_for_bit(own_stream):
    """the weight gradients' side stream against the chain it runs beside"""
    from lbm_mirror_gb300 import UNet
    h, w, n = 32, 128, 2
    gen = torch.Generator().manual_seed(5)
    net = UNet(height=h, width=w, widths=(32, 64, 64, 128), out_channels=3, max_batch=n, seed=3)
    stream = torch.cuda.Stream()
    if not own_stream:
        net.set_stream(stream.cuda_stream)
    x = torch.randn((n, h, w, 16), generator=gen).to(torch.bfloat16).cuda()
    t = torch.randn((n, h, w, 3), generator=gen).cuda()
    torch.cuda.synchronize()
    net.set_input(x.data_ptr(), n)
    net.forward(n)
    first = None
    for _ in range(20):
        net.backward(t.data_ptr(), n)
        g = net.grads()
        first = g if first is None else first
        assert np.array_equal(g, first)
