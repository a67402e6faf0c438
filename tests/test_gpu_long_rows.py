"""One-column kernel on rows longer than a model's, where the expanded grids of IQ2 / IQ1 no longer fit beside the column
and the 16-bit codes (in tiles of eight, four and two rows) take over.  Against torch in 64 bits on the exact weights and
the Q8_K values: the integer sums are exact, a row's fp32 sum has one product per 32 weights (three roundings), five
butterfly additions and one addition per slice of 1024 weights, each within 2^-24 of what it adds up."""
import pytest
import torch

from qwengine_b200 import api, formats as F, synth

pytestmark = pytest.mark.gpu
LONGEST = {"IQ2_XXS": 137216, "IQ2_XS": 148480, "IQ2_S": 144384, "IQ1_S": 145408, "IQ1_M": 141312}


@pytest.mark.parametrize("name", sorted(LONGEST))
@pytest.mark.parametrize("K", [30720, 65536, 98304, 0])
def test_long_rows(ctx, name, K):
    f, M, nb = F.get(name), 41, 2
    K = K or LONGEST[name]
    w = torch.from_numpy(synth.make_weights(f, M, K, seed=K)).cuda()
    x = torch.from_numpy(synth.make_activations(nb, K, seed=8)).cuda()
    xq = ctx.quantize_q8k(x)
    y = ctx.gemv(f, w, xq, K)
    ctx.check()
    blocks = xq.view(nb, K // 256, F.Q8K_BLOCK_BYTES)
    d = blocks[:, :, :4].contiguous().view(torch.float32).double()
    xv = (blocks[:, :, 4:260].contiguous().view(torch.int8).double() * d).view(nb, K)
    wd = ctx.dequant_rows(f, w, K, kind=api.OUT_F32).double()
    ref, mag = xv @ wd.t(), xv.abs() @ wd.abs().t()
    assert float(((y.double() - ref).abs() / mag).max()) < (K / 1024 + 8) * 2.0 ** -24
    one = torch.cat([ctx.gemv(f, w, xq[c:c + 1], K) for c in range(nb)])
    assert torch.equal(one.view(torch.int32), y.view(torch.int32))
