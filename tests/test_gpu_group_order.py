"""A group's run starts after what its contexts' own streams hold."""
import re
from pathlib import Path

import numpy as np
import pytest

API = Path(__file__).resolve().parents[1] / "cdixx_gb300" / "csrc" / "cdx_api.cu"


def test_group_waits_for_its_contexts_streams():
    body = re.search(r"int group_run_impl\(.*?\n}\n", API.read_text(), re.S).group(0)
    launch = body.index("cudaGraphLaunch(")
    after_capture = body.index("g->gkey = key;")
    assert "cudaStreamWaitEvent(g->st" in body[after_capture:launch]


@pytest.mark.gpu
@pytest.mark.parametrize("concurrent", [False, True])
def test_group_run_follows_asynchronous_runs(cdx, torch_cuda, concurrent):
    torch = torch_cuda
    sizes, first, second = ((1024, 2), (512, 8)), "2*shrinkWrap+300*HIO", "1*shrinkWrap+20*RAAR"
    g = torch.Generator(device="cuda").manual_seed(4)
    pats = [torch.poisson(torch.rand(n, n, device="cuda", generator=g) ** 8 * 6, generator=g) for n, _ in sizes]
    torch.cuda.synchronize()   # the contexts read them on streams of their own
    out = []
    for asynchronous in (False, True):
        ctxs = [cdx.Context(cdx.default_params(n, n, batch=b, beta=0.9, shrink_threshold=0.1)) for n, b in sizes]
        for c, p, (_, b) in zip(ctxs, pats, sizes):
            for k in range(b):
                c.set_pattern(k, p)
            c.random_start(6)
        grp = cdx.Group(ctxs, concurrent=concurrent)
        grp.run(second)   # captured before
        for c in ctxs:
            c.random_start(6)
            (c.run_async if asynchronous else c.run)(first)
        grp.run(second)
        out.append([(c.get_object(b - 1), c.get_support(b - 1)) for c, (_, b) in zip(ctxs, sizes)])
        grp.close()
        for c in ctxs:
            c.close()
    for (a, s), (b, t) in zip(*out):
        assert np.array_equal(a, b) and np.array_equal(s, t) and np.isfinite(a).all()


@pytest.mark.gpu
def test_group_run_takes_a_beamstop_set_after_a_run(cdx, torch_cuda):
    """A beamstop given after the group captured the algorithm is in its next run, as in a context's."""
    torch = torch_cuda
    n = 128
    g = torch.Generator(device="cuda").manual_seed(8)
    pat = torch.poisson(torch.rand(n, n, device="cuda", generator=g) ** 8 * 6, generator=g)
    stop = (torch.rand(n, n, device="cuda", generator=g) > 0.7).float()
    torch.cuda.synchronize()   # the contexts read them on streams of their own
    p = cdx.default_params(n, n, beta=0.9, sim_ccd_bit=1, noise_level=4, exposure=0.1)
    out = []
    for grouped in (False, True):
        with cdx.Context(p) as ctx:
            owner = cdx.Group([ctx]) if grouped else ctx
            ctx.set_pattern(0, pat)
            for given in (False, True):
                if given:
                    ctx.set_beamstop(0, stop)
                ctx.random_start(3)
                owner.run("5*RAAR")
                out.append(ctx.get_object(0))
            if grouped:
                owner.close()
    assert np.array_equal(out[0], out[2]) and np.array_equal(out[1], out[3])
    assert not np.array_equal(out[0], out[1])
