"""Top-k where its lists and candidate counts can go wrong: one logit, chunks of 1024 with one missing or one over, exactly
and one list more than the candidates of the smaller merge, the largest vector; few distinct values (ties within and
across chunks decide), the lowest finite values and NaN."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 131072, 131073, 393216])
@pytest.mark.parametrize("k", [1, 64])
@pytest.mark.parametrize("kind", ["normal", "ties", "low"])
def test_edges(ctx, n, k, kind):
    rng = np.random.default_rng(n + k)
    x = rng.standard_normal((2, n)).astype(np.float32)
    if kind == "ties":
        x = rng.integers(-1, 2, size=(2, n)).astype(np.float32)
    elif kind == "low":
        x = rng.choice(np.array([np.finfo(np.float32).min, -np.inf, np.nan, -0.0], np.float32), size=(2, n), p=[0.00005, 0.49995, 0.49995, 0.00005])
    vals, idx = ctx.topk(torch.from_numpy(x).cuda(), k)
    ctx.check()
    want_v, want_i = oracle.topk(x, k)
    assert np.array_equal(idx.cpu().numpy(), want_i)
    assert np.array_equal(vals.cpu().numpy().view(np.uint32), want_v.view(np.uint32))
