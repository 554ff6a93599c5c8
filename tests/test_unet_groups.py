"""Channels of a GroupNorm group: at most 256 at the deepest level.  More are refused by
cdx_unet_create before it looks for a device (the statistics kernels would not end)."""
import ctypes

import numpy as np
import pytest


@pytest.mark.parametrize("base,groups,levels,ok", [
    (64, 1, 4, False), (32, 8, 8, False), (256, 1, 2, False), (64, 1, 3, True), (32, 8, 7, True), (256, 2, 2, True)])
def test_group_channels_are_bounded(cdx, base, groups, levels, ok):
    from cdixx_gb300 import unet
    cfg = unet.default_config(n=8 << levels, levels=levels, base=base, groups=groups, batch=0)   # a batch of 0 is refused last
    with pytest.raises(cdx.CdxError) as e:
        cdx.check(cdx.lib().cdx_unet_create(ctypes.byref(cfg), None, ctypes.byref(ctypes.c_void_p())))
    assert e.value.code == cdx.CDX_ERR_ARG
    assert ("256 channels" in str(e.value)) == (not ok) and ("batch" in str(e.value)) == ok


@pytest.mark.gpu
def test_largest_groups_match_oracle(cdx, torch_cuda):
    """Groups of 256 channels, with the bounds of test_gpu_unet.py."""
    from cdixx_gb300 import unet
    from oracle import unet_oracle as U
    from tests.test_gpu_unet import small_case
    torch = torch_cuda
    n, levels, base, groups, batch = 32, 3, 64, 1, 2
    I, amp, ph, sup = small_case(n, batch, seed=6)
    p = U.init_params(n, levels, base, seed=13)
    loss_ref, g_ref, out_ref = U.forward_backward(p, I, amp, ph, sup, n, levels, base, groups=groups, round_bf16=True)
    with unet.UNet(n=n, levels=levels, base=base, batch=batch, groups=groups) as net:
        net.set_params(p)
        dev = [torch.from_numpy(x).cuda() for x in (I, amp, ph, sup)]
        out = net.forward(dev[0]).cpu().numpy().transpose(0, 2, 3, 1)
        loss = net.loss_backward(*dev)
        g = net.grads().astype(np.float64)
    rel = lambda a, b: np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)
    assert rel(out, out_ref) < 5e-3
    assert abs(loss - loss_ref) <= 2e-3 * abs(loss_ref)
    assert rel(g, g_ref) < 3e-2
