"""Pairs of CTAs of which one finishes first: with an odd number of row tiles the last pair's second half stores nothing, while the
first still reads its accumulators, which belong to an allocation of both.  Two accumulators of 256 tokens into rows that are added to
(the slowest way out) and one super-block (the shortest way in), several times over, checked as the other cuts are."""
import pytest
import torch

from test_gpu_prefill_cuts import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["Q8_0", "Q4_K", "IQ2_XS"])
@pytest.mark.parametrize("M,K,B", [(100, 256, 512), (260, 256, 512), (640, 512, 1000), (385, 256, 258)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_a_half_without_rows(ctx, name, M, K, B, dt):
    for _ in range(4):
        check(ctx, name, M, K, B, dt, (B + 511) // 512, 1, accumulate=True)
