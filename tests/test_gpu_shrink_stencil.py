"""The shrinkwrap stencils at every radius regime (none, fewer taps than a thread's outputs,
around that, large, capped by the size) and at sizes below a CTA's rows or a warp's columns:
the support field of the |rho|^2 mode against the periodic convolution in float64.  All terms
are non-negative, so the relative error is bounded by the number of roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [0.3, 0.4, 1.0, 1.4, 2.7, 10.0, 30.0])
@pytest.mark.parametrize("rows,cols,batch", [(16, 16, 2), (24, 96, 1), (64, 256, 3), (192, 384, 1), (512, 32, 2)])
def test_support_field(cdx, rows, cols, batch, sigma):
    rng = np.random.default_rng(rows + cols)
    p = cdx.default_params(rows, cols, batch=batch, shrink_mode=cdx.SHRINK_SPATIAL, sigma0=sigma, shrink_threshold=0.1)
    with cdx.Context(p) as ctx:
        for k in range(batch):
            ctx.set_pattern(k, rng.random((rows, cols)).astype(np.float32))
        ctx.random_start(4)
        ctx.run("1*HIO+1*shrinkWrap")
        for k in range(batch):
            v = np.abs(ctx.get_object(k).astype(np.complex128)) ** 2 / (rows * cols)
            taps = 0
            for ax, n in enumerate((rows, cols)):
                r = max(0, min(int(np.floor(np.float32(sigma) * 6)) >> 1, (n - 1) // 2, 64))
                w = np.exp(-np.arange(-r, r + 1) ** 2 / (2.0 * float(np.float32(sigma)) ** 2))
                w /= w.sum()
                v = sum(wi * np.roll(v, d, ax) for d, wi in zip(range(-r, r + 1), w))
                taps += 2 * r + 1
            got = ctx.get_support(k)
            # products, weights and sums of both passes, |rho|^2 and its scale
            assert np.all(np.abs(got - v) <= (2 * taps + 12) * 2.0 ** -24 * v)
