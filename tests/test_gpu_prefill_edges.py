"""Prefill around the line between operand A in tensor memory (up to 256 tokens) and in shared memory: every format, rows that
start only 2 bytes aligned and are padded, single and ragged rows (the unchecked fetch stops short of the matrix's first and
last unit), one to four super-blocks.  Bound per output: weights, activations' products and, for the packed K-quants, scales
rounded to 8 bits (2^-9 each, two of them), fp32 sums: 2^-7 of the sum of |w x| is twice that."""
import pytest
import torch

from qwengine_b200 import formats as F, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", sorted(F.ALL_FORMATS))
@pytest.mark.parametrize("M,K,B,pad,shift", [(1, 256, 16, 0, 0), (129, 512, 256, 0, 0), (131, 768, 257, 6, 2), (257, 1024, 33, 2, 2), (128, 1280, 241, 16, 0)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_rows_and_tokens(ctx, name, M, K, B, pad, shift, dt):
    f = F.get(name)
    rb = f.row_bytes(K) + pad
    buf = torch.full((M * rb + 64,), 0x5A, dtype=torch.uint8, device="cuda")
    w = buf[shift:shift + M * rb].view(M, rb)
    packed = torch.from_numpy(synth.make_weights(f, M, K, seed=M + K, scale=1e-3)).cuda()
    w[:, :f.row_bytes(K)].copy_(packed)
    x = torch.randn((B, K), device="cuda", generator=torch.Generator("cuda").manual_seed(B)).to(dt)
    got = ctx.gemm_prefill(f, w, x, K).double()
    ctx.check()
    wd = ctx.dequant_rows(f, packed, K).double()
    want, mag = x.double() @ wd.T, x.double().abs() @ wd.abs().T
    assert bool(((got - want).abs() <= 2.0 ** -7 * mag + 1e-6).all())
