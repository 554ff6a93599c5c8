"""Batches that outgrow the L2 run in chunks between shrinkwraps: every pattern ends with the
bits, R-factors and stops it gets alone, with even and uneven chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,batch,ccd", [(512, 512, 26, 0), (512, 512, 51, 0), (768, 512, 18, 1), (2048, 2048, 2, 0)])
@pytest.mark.parametrize("stops", [True, False])
def test_chunked_batch_equals_alone(cdx, torch_cuda, rows, cols, batch, ccd, stops):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(batch)
    base = torch.rand(rows, cols, device="cuda", generator=g) ** 8
    kw = dict(beta=0.9, shrink_threshold=0.1, rf_every=2)
    if stops:   # these runs stay whole
        kw.update(stop_rfactor=0.4, plateau_iters=6)
    if ccd:
        kw.update(sim_ccd_bit=1, noise_level=4, exposure=0.1)
    inten = [torch.poisson(base * (2 + 5 * k), generator=g) for k in range(batch)]
    psi0 = [torch.polar(i.sqrt(), 6.28 * torch.rand(rows, cols, device="cuda", generator=g)).contiguous() for i in inten]
    torch.cuda.synchronize()   # the contexts read these on streams of their own
    algo = "4*RAAR+1*shrinkWrap+9*ER+1*shrinkWrap+3*HIO"
    assert 20 * rows * cols * batch > 125e6

    def run(which):
        with cdx.Context(cdx.default_params(rows, cols, batch=len(which), **kw)) as ctx:
            for j, k in enumerate(which):
                ctx.set_pattern(j, inten[k])
                ctx.set_initial(j, psi0[k])
            ctx.run(algo)
            keys = ("rfactor", "rfactor_min", "converged_iter", "threshold", "flags", "residual")
            return [(ctx.get_object(j), ctx.get_support(j), [ctx.stats(j)[s] for s in keys]) for j in range(len(which))]

    whole = run(range(batch))
    for k in (0, batch // 2 - 1, batch // 2, batch - 1):
        alone = run([k])[0]
        assert np.array_equal(whole[k][0], alone[0]) and np.array_equal(whole[k][1], alone[1])
        assert whole[k][2] == alone[2], k
