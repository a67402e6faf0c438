"""Top-k around the number of elements that are picked one by one: vectors shorter than k, chunks of 1024 with one missing
or one over, the most chunks; ties within and across chunks, the lowest values and NaN."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5, 1023, 1025, 131073, 393216])
@pytest.mark.parametrize("kind", ["normal", "ties", "low"])
def test_few(ctx, n, kind):
    for k in (1, 2, 3, 7, 8, 9, 12, 15, 16, 17):
        rng = np.random.default_rng(n + k)
        if kind == "normal":
            x = rng.standard_normal((2, n)).astype(np.float32)
        elif kind == "ties":
            x = rng.integers(-1, 2, size=(2, n)).astype(np.float32)
        else:
            p = [4 / n, 0.5 - 4 / n, 0.5 - 4 / n, 4 / n] if n > 100 else [0.25] * 4
            x = rng.choice(np.array([np.finfo(np.float32).min, -np.inf, np.nan, -0.0], np.float32), size=(2, n), p=p)
        vals, idx = ctx.topk(torch.from_numpy(x).cuda(), k)
        ctx.check()
        want_v, want_i = oracle.topk(x, k)
        assert np.array_equal(idx.cpu().numpy(), want_i), k
        assert np.array_equal(vals.cpu().numpy().view(np.uint32), want_v.view(np.uint32)), k
