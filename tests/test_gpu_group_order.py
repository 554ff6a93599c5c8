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
