"""A context or group that is given stops after it ran an algorithm runs it as one that had
them from the start (whole, not in chunks), and as before once they are taken back: the
launch counts of the captured graphs say which."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, BATCH = 512, 26
ALGO = "1*shrinkWrap+5*HIO"


def fill(ctx, inten):
    for k in range(BATCH):
        ctx.set_pattern(k, inten)
    ctx.random_start(2)


@pytest.mark.parametrize("group", [False, True])
def test_stops_set_after_a_run(cdx, torch_cuda, group):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(3)
    inten = torch.poisson(torch.rand(N, N, device="cuda", generator=g) ** 8 * 6, generator=g)
    torch.cuda.synchronize()   # the contexts read it on streams of their own
    p = cdx.default_params(N, N, batch=BATCH, beta=0.9, rf_every=2)

    def run(ctx, owner):
        fill(ctx, inten)
        owner.run(ALGO)
        return ctx.stats(0)["launches"], ctx.get_object(BATCH - 1)

    with cdx.Context(p) as ctx:   # stops from the start
        ctx.set_stop_rfactor(1, 1e-12)
        whole, ref = run(ctx, ctx)
    with cdx.Context(p) as ctx:
        owner = cdx.Group([ctx]) if group else ctx
        chunked, a = run(ctx, owner)
        assert chunked > whole
        ctx.set_stop_rfactor(1, 1e-12)
        again, b = run(ctx, owner)
        ctx.set_stop_rfactor(1, 0.0)
        back, c = run(ctx, owner)
        if group:
            owner.close()
    assert again == whole and back == chunked
    assert all(np.array_equal(ref, x) for x in (a, b, c))
