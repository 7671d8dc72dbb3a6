"""The gradient kernel at the edges of its tiles (128 samples) and of its grid (one block per
multiprocessor, so two to three tiles per block), and the weights' operand images after Adam steps.

Gradient tolerance: as in test_gpu_mlp.py, 1e-2 in relative L2 norm per parameter tensor (the SiLU's
hardware tanh, about 2^-11 per activation, and the BF16 roundings it moves)."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo
from test_gpu_mlp import _problem, net  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", [1, 127, 129, "1", "2-", "2+"])
def test_gradient_at_tile_and_grid_edges(net, where):  # noqa: F811
    import torch

    if isinstance(where, str):
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        n = int(where[0]) * 128 * sms + {"": 1, "-": -1, "+": 1}[where[1:]]
    else:
        n = where
    params, mean, inv_std, scale, feat, target = _problem(9, n)
    net.set_params(params)
    net.set_normalization(mean, inv_std, scale)
    f, t = torch.from_numpy(feat).cuda(), torch.from_numpy(target).cuda()
    g, loss = net.gradient(f, t)
    again, loss2 = net.gradient(f, t)  # the accumulators start from zero again
    norm = np.concatenate([mean, inv_std, [scale, 1.0]])
    gw, lw = mo.gradient(params, norm, feat, target, emulate=True)
    assert abs(loss - lw) <= 1e-2 * lw and abs(loss2 - loss) <= 1e-5 * abs(loss)
    got, want, rep = mo.unpack(g), mo.unpack(gw), mo.unpack(again)
    for name, _ in mo.SIZES:
        r = np.linalg.norm(want[name])
        assert np.linalg.norm(got[name] - want[name]) <= 1e-2 * r + 1e-9, name
        # two runs differ by the order of their FP32 additions alone
        assert np.linalg.norm(got[name] - rep[name]) <= 1e-5 * r + 1e-9, name


def test_images_follow_adam_steps(net):  # noqa: F811
    """The forward pass reads the weights' BF16 images, which Adam steps update in place: the same
    outputs as a network that is given the updated parameters anew."""
    import torch

    from akuaengine_gb300.warm_start import LambdaNet

    params, mean, inv_std, scale, feat, target = _problem(4, 1000)
    net.set_params(params)
    net.set_normalization(mean, inv_std, scale)
    f, t = torch.from_numpy(feat).cuda(), torch.from_numpy(target).cuda()
    for _ in range(3):
        net.adam_step(f, t, 1e-2)
    now = net.params()
    assert np.abs(now - params).max() > 1e-3
    fresh = LambdaNet(now)
    try:
        fresh.set_normalization(mean, inv_std, scale)
        assert torch.equal(net.forward(f), fresh.forward(f))
        assert fresh.gradient(f, t)[1] == pytest.approx(net.gradient(f, t)[1], rel=1e-5)
    finally:
        fresh.close()


@pytest.mark.parametrize("rounds", [1, 4, 5])
def test_forward_grid_edges(net, rounds):  # noqa: F811
    """Counts around a tile for every block (two per multiprocessor), for every warpgroup of them, and
    beyond: a sample's output does not depend on the others, so it equals that of a small call bit
    for bit."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    params, mean, inv_std, scale, feat, _ = _problem(6, 128 * 2 * sms * rounds + 1)
    net.set_params(params)
    net.set_normalization(mean, inv_std, scale)
    f = torch.from_numpy(feat).cuda()
    for n in (len(feat), len(feat) - 2):
        want = torch.cat([net.forward(f[k:min(k + 8000, n)]) for k in range(0, n, 8000)])
        assert torch.equal(net.forward(f[:n]), want)
