"""The training gradient over batches that give its persistent CTAs none, one
or two tiles of 128 samples more than their neighbours: against the oracle
with the kernel's roundings (its 2e-2, normwise per parameter group), and
the same samples in another order of tiles, which only reorders FP32 sums:
at most 1200 partial sums, each addition off by 2^-24 of the running sum at
most (1200 * 2^-24 = 7e-5 normwise)."""
import numpy as np
import pytest

from oracle import mlp_oracle

pytestmark = pytest.mark.gpu


def _data(tiles):
    import torch
    g = torch.Generator(device="cuda").manual_seed(tiles)
    n = 128 * tiles
    x = torch.randn((n, 48), generator=g, device="cuda")
    x[:, 45:] = 0.0
    return x.to(torch.bfloat16), torch.randn((n, 2), generator=g, device="cuda")


@pytest.mark.parametrize("tiles", [1, 2, 147, 295, 296, 297, 592, 593, 1185])
def test_gradient_does_not_depend_on_the_order_of_tiles(gpu, tiles):
    import torch
    from inmsom_elfs_b200.mlp import MLP
    x, t = _data(tiles)
    net = MLP(seed=tiles)
    idx = torch.arange(128 * tiles, device="cuda", dtype=torch.int32)
    want = net.loss_grad(x, t).cpu().numpy()
    assert np.array_equal(want, net.loss_grad(x, t, idx).cpu().numpy())
    for shift in (1, 2, 148, 296):
        got = net.loss_grad(x, t, torch.roll(idx, 128 * shift)).cpu().numpy()
        for a, b in ((got[:-1], want[:-1]), (got[-1:], want[-1:])):
            assert np.abs(a - b).max() <= 7e-5 * np.abs(b).max(), shift


@pytest.mark.parametrize("tiles", [1, 3, 297])
def test_gradient_matches_oracle(gpu, tiles):
    from inmsom_elfs_b200.mlp import MLP
    x, t = _data(tiles)
    net = MLP(seed=tiles)
    got = net.loss_grad(x, t).cpu().numpy().astype(np.float64)
    loss, want = mlp_oracle.loss_grad(net.host_params(), x.float().cpu().numpy(), t.cpu().numpy())
    assert abs(got[-1] - loss) <= 2e-2 * loss
    o = mlp_oracle
    cuts = (o.OFF_W1, o.OFF_B1, o.OFF_W2, o.OFF_B2, o.OFF_W3, o.OFF_B3, o.NPARAM)
    for a, b in zip(cuts[:-1], cuts[1:]):
        assert np.abs(got[a:b] - want[a:b]).max() <= 2e-2 * np.abs(want[a:b]).max(), (a, b)


@pytest.mark.parametrize("rows", [1, 15, 64, 65, 4099])
def test_forward_wherever_the_weights_start(gpu, rows):
    """Weights read 16 bytes at a time where they start on 16 bytes, one by
    one elsewhere: the same values, and the oracle's within the 2e-3 of the
    hardware tanh (2^-11) and the BF16 activations."""
    import torch
    from inmsom_elfs_b200 import _lib
    from inmsom_elfs_b200.mlp import MLP
    every = _data(33)[0]
    x = every[:rows].contiguous()
    net = MLP(seed=rows)
    want = net.forward(x).cpu().numpy()
    y, _ = mlp_oracle.forward(net.host_params(), every.float().cpu().numpy(), emulate=True)
    assert np.abs(want - y[:rows]).max() <= 2e-3 * np.abs(y).max()
    room = torch.empty(_lib.MLP_NBF16 + 8, dtype=torch.bfloat16, device="cuda")
    for off in (1, 4, 7):
        net2 = MLP(net.host_params())
        net2.wbf16 = room[off:off + _lib.MLP_NBF16].copy_(net.wbf16)
        assert np.array_equal(net2.forward(x).cpu().numpy(), want), off
