"""Statistics asked for by several threads at once: each gets those of its own pattern."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_stats_from_several_threads(cdx, torch_cuda):
    n, batch = 64, 4
    rng = np.random.default_rng(5)
    with cdx.Context(cdx.default_params(n, n, batch=batch, beta=0.9)) as ctx:
        for k in range(batch):
            ctx.set_pattern(k, (rng.random((n, n)) * (1 + k)).astype(np.float32))
        ctx.random_start(1)
        ctx.run("3*HIO")
        want = [ctx.stats(k)["residual"] for k in range(batch)]
        assert len(set(want)) == batch
        wrong = [0] * batch

        def ask(k):
            for _ in range(4000):
                wrong[k] += ctx.stats(k)["residual"] != want[k]

        threads = [threading.Thread(target=ask, args=(k,)) for k in range(batch)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert wrong == [0] * batch
