"""A training step after kel_unet_set_residual or kel_unet_set_conv_kernel runs
the new setting, also where the step before it replayed a captured graph: loss
and gradients are bit for bit those of forward and backward calls on a net that
never captured anything, for the first step after the change and for the one
that replays its new capture."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

H, W, N = 16, 128, 2

CHANGES = {
    "residual": lambda net: net.set_residual(0, 1, 2.0),
    "residual scale": lambda net: net.set_residual(2, 2, -0.5),
    "residual off": lambda net: net.set_residual(-1),
    "mma_sync": lambda net: net.set_conv_kernel(1),
}


@pytest.mark.parametrize("change", list(CHANGES))
def test_a_step_runs_the_setting_of_its_call(change):
    from lbm_mirror_gb300 import UNet
    rng = np.random.default_rng(5)
    x = torch.tensor(rng.standard_normal((N, H, W, 16)), dtype=torch.bfloat16, device="cuda")
    target = torch.tensor(rng.standard_normal((N, H, W, 3)), dtype=torch.float32, device="cuda")
    nets = [UNet(height=H, width=W, widths=(16, 32, 32, 48), max_batch=N, seed=3) for _ in range(2)]
    start = nets[0].params()
    torch.cuda.synchronize()

    def prepare(net, step):
        net.set_params(start)
        net.set_input(x.data_ptr(), N)
        if step == 0:
            net.set_residual(2, 2, 1.0)
        if step == 3:
            CHANGES[change](net)

    results = []
    for net, captured in zip(nets, (True, False)):
        out = []
        for step in range(6):  # 0 one by one, 1 captures, 2 replays; the change; 3 .. 5 the same again
            prepare(net, step)
            if captured:
                net.train_step(target.data_ptr(), N)
                loss = net.last_loss()
            else:
                net.forward(N)
                loss = net.backward(target.data_ptr(), N)
                net.synchronize()
            out.append((loss, net.grads()))
        results.append(out)
        net.close()
    for step, ((la, ga), (lb, gb)) in enumerate(zip(*results)):
        assert la == lb, (step, la, lb)
        np.testing.assert_array_equal(ga, gb, err_msg=f"gradients of step {step}")
    assert not np.array_equal(results[1][2][1], results[1][3][1])  # the change shows
