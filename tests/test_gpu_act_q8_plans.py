"""One column with per-32 activations runs with one or two CTAs per SM, by format and row length: the same bits either way."""
import pytest
import torch

from qwengine_b200 import formats as F, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", list(F.ALL_FORMATS))
def test_either_plan_gives_the_same_bits(ctx, name):
    f, M = F.get(name), 77
    for K in (256, 1024, 2048, 2304, 3072, 3328, 4096, 4352, 5120, 6144, 6400, 8192, 13312, 14336, 17408):
        w = torch.from_numpy(synth.make_weights(f, M, K, seed=K)).cuda()
        q, d, _ = ctx.quantize_act_q8(torch.from_numpy(synth.make_activations(1, K, seed=9)).cuda())
        got = ctx.gemv_act_q8(f, w, q, d, K)
        ctx.debug_set_one_cta(0)
        try:
            two = ctx.gemv_act_q8(f, w, q, d, K)
        finally:
            ctx.debug_set_one_cta(1)
        assert torch.equal(got.view(torch.int32), two.view(torch.int32)), (name, K)
    ctx.check()
