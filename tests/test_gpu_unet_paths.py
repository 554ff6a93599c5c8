"""The U-Net's kernels against one another: the tcgen05 patch convolutions and row-segment weight
gradients (umma 0 and 1, where a layer fits them), the gathering tcgen05 convolutions and the
mma.sync kernels (umma 3 and 2, for every layer) give the same bits in outputs, loss and
gradients, and layers of more than 256 channels match the oracle."""
import numpy as np
import pytest

from oracle import unet_oracle as U
from tests.test_gpu_unet import small_case

pytestmark = pytest.mark.gpu


def results(torch, cfg, p, case, mode):
    from cdixx_gb300 import unet
    with unet.UNet(umma=mode, **cfg) as net:
        net.set_params(p)
        dev = [torch.from_numpy(x).cuda() for x in case]
        out = net.forward(dev[0]).cpu().numpy()
        loss = net.loss_backward(*dev)
        return out, loss, net.grads()


@pytest.mark.parametrize("n,levels,base,batch", [
    (16, 2, 16, 1),      # grids smaller than a tile, weight-gradient rows of 16 and 8 pixels
    (96, 3, 16, 2),      # half-filled last tiles, odd multiples of 16 a row
    (48, 2, 24, 3),      # channels that are no whole 16s at the first level
    (64, 3, 32, 5),      # resident and streamed weights, stride 2, transposed layers, skips
    (64, 4, 64, 1),      # 512 channels at the deepest level
    (256, 2, 32, 5),     # a forward pass that launches dependently, and whole segments of 256 pixels
])
def test_kernels_agree(cdx, torch_cuda, n, levels, base, batch):
    p = U.init_params(n, levels, base, seed=21)
    case = small_case(n, batch, seed=8)
    cfg = dict(n=n, levels=levels, base=base, batch=batch, groups=3 if base == 24 else 8)
    ref = results(torch_cuda, cfg, p, case, 2)
    assert np.isfinite(ref[0]).all() and np.isfinite(ref[2]).all() and np.any(ref[2])
    for mode in (0, 1, 3):
        out, loss, grads = results(torch_cuda, cfg, p, case, mode)
        assert np.array_equal(out, ref[0]) and loss == ref[1] and np.array_equal(grads, ref[2]), mode


@pytest.mark.parametrize("mode", [0, 1])
def test_wide_layers_match_oracle(cdx, torch_cuda, mode):
    """256 and 512 channels, with the bounds of test_gpu_unet.py."""
    n, levels, base, batch = 32, 3, 128, 1
    case = small_case(n, batch, seed=12)
    p = U.init_params(n, levels, base, seed=17)
    loss_ref, g_ref, out_ref = U.forward_backward(p, *case, n, levels, base, round_bf16=True)
    out, loss, g = results(torch_cuda, dict(n=n, levels=levels, base=base, batch=batch), p, case, mode)
    rel = lambda a, b: np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)
    assert rel(out.transpose(0, 2, 3, 1), out_ref) < 5e-3
    assert abs(loss - loss_ref) <= 2e-3 * abs(loss_ref)
    assert rel(g.astype(np.float64), g_ref) < 3e-2
