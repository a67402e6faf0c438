"""Prefill by pairs of CTAs (more than 256 tokens, K not shared): an odd number of row tiles, whose last pair has a half without
rows, ragged rows, the smallest and largest token tiles, a last tile shorter than half of one, one super-block.  Bound per
output as around the other operand layouts: 2^-9 for the weight and 2^-9 for packed scales, doubled, of the sum of |w x|."""
import pytest
import torch

from qwengine_b200 import formats as F, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", sorted(F.ALL_FORMATS))
@pytest.mark.parametrize("M,K,B,tiles,shift", [(129, 256, 257, 1, 0), (257, 512, 512, 1, 2), (383, 1280, 300, 1, 0), (256, 768, 1025, 3, 0), (130, 1024, 545, 2, 2)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_pairs(ctx, name, M, K, B, tiles, shift, dt):
    f = F.get(name)
    rb = f.row_bytes(K) + shift
    buf = torch.full((M * rb + 64,), 0x5A, dtype=torch.uint8, device="cuda")
    w = buf[shift:shift + M * rb].view(M, rb)
    packed = torch.from_numpy(synth.make_weights(f, M, K, seed=M + K, scale=1e-3)).cuda()
    w[:, :f.row_bytes(K)].copy_(packed)
    x = torch.randn((B, K), device="cuda", generator=torch.Generator("cuda").manual_seed(B)).to(dt)
    assert ctx.lib.q38b_debug_set_prefill_cut(ctx.h, tiles, 1) == 0
    try:
        got = ctx.gemm_prefill(f, w, x, K).double()
        ctx.check()
    finally:
        ctx.lib.q38b_debug_set_prefill_cut(ctx.h, 0, 0)
    wd = ctx.dequant_rows(f, packed, K).double()
    want, mag = x.double() @ wd.T, x.double().abs() @ wd.abs().T
    assert bool(((got - want).abs() <= 2.0 ** -7 * mag + 1e-6).all())
