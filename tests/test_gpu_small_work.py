"""The geometry for small work (lengths of 1024 up to 2^21 pixels) against the general one:
a pattern alone and the same pattern in a batch past the limit give the same bits, for
square and oblong shapes, both projections and the common updates."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ccd", [0, 1])
@pytest.mark.parametrize("rows,cols,batch", [(1024, 1024, 3), (1024, 384, 6), (256, 1024, 9), (1024, 16, 129),
                                             (1024, 2048, 2)])
def test_alone_and_in_a_batch(cdx, torch_cuda, rows, cols, batch, ccd):
    torch = torch_cuda
    assert rows * cols <= 1 << 21 < rows * cols * batch
    g = torch.Generator(device="cuda").manual_seed(rows + 3 * cols)
    inten = torch.poisson(torch.rand(rows, cols, device="cuda", generator=g) ** 8 * 6, generator=g)
    psi0 = torch.polar(inten.sqrt(), 6.28 * torch.rand(rows, cols, device="cuda", generator=g)).contiguous()
    torch.cuda.synchronize()   # the contexts read these on streams of their own
    kw = dict(sim_ccd_bit=1, noise_level=4, exposure=0.1) if ccd else {}
    out = []
    for b in (1, batch):
        with cdx.Context(cdx.default_params(rows, cols, batch=b, beta=0.9, shrink_threshold=0.1, **kw)) as ctx:
            for k in range(b):
                ctx.set_pattern(k, inten)
                ctx.set_initial(k, psi0)
            ctx.run("2*HIO+1*shrinkWrap+2*RAAR+2*ER")
            out.append((ctx.get_object(b - 1), ctx.get_fourier(b - 1), ctx.get_support(b - 1)))
    for x, y in zip(*out):
        assert np.array_equal(x, y)
