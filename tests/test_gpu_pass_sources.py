"""A recorded pass equals the calls whatever buffer its columns come from: columns that start at an odd float."""
import pytest
import torch

from qwengine_b200 import Pass, formats as F, synth

pytestmark = pytest.mark.gpu


def weights(f, M, K):
    return torch.from_numpy(synth.make_weights(f, M, K, seed=M + K)).cuda()


def same(a, b):
    return torch.equal(a.contiguous().view(torch.int32), b.contiguous().view(torch.int32))


@pytest.mark.parametrize("name", ["IQ2_S", "Q2_K", "Q4_K", "IQ3_XXS"])
@pytest.mark.parametrize("nb", range(1, 9))
def test_source_of_odd_length(ctx, name, nb):
    f, K, M1, M2 = F.get(name), 2816, 130, 77
    w1, w2 = weights(f, M1, K), weights(f, M2, K)
    x = torch.from_numpy(synth.make_activations(nb, K, seed=6)).cuda()
    ps = Pass(ctx, max_nb=nb)
    xin, xq, y = ps.buffer_f32(K + 1), ps.buffer_q8k(K), ps.buffer_f32(M1 + M2)
    ps.quantize(xin, 0, K, xq)
    ps.gemv(ps.matrix_device(f, w1, K), xq, y, 0)
    ps.gemv(ps.matrix_device(f, w2, K), xq, y, M1)
    ps.buffer_tensor(xin)[:, :K].copy_(x)
    ps.run(nb)
    torch.cuda.synchronize()
    ctx.check()
    got = ps.buffer_tensor(y).clone()
    ps.close()
    xq8 = ctx.quantize_q8k(x)
    assert same(got[:, :M1], ctx.gemv(f, w1, xq8, K)) and same(got[:, M1:], ctx.gemv(f, w2, xq8, K))
