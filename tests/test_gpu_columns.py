"""Two to eight columns on the one-column kernel's arithmetic (the formats without mma fragments, the per-32 activations):
every column is the single call's result bit for bit, whatever launches it shares, for rows of one to 17 slices (the last
one ragged), ragged tiles, output strides and accumulation; and a recorded pass equals the calls."""
import pytest
import torch

from qwengine_b200 import Pass, formats as F, synth

pytestmark = pytest.mark.gpu
ONE_COLUMN = ["Q2_K", "IQ2_XXS", "IQ2_XS", "IQ2_S", "IQ1_S", "IQ1_M"]
SHAPES = [(1, 256), (7, 1280), (333, 2816), (1500, 5120), (40, 17408)]


def weights(f, M, K):
    return torch.from_numpy(synth.make_weights(f, M, K, seed=M + K)).cuda()


def same(a, b):
    return torch.equal(a.contiguous().view(torch.int32), b.contiguous().view(torch.int32))


@pytest.mark.parametrize("name", ONE_COLUMN)
@pytest.mark.parametrize("M,K", SHAPES)
def test_gemv_columns_are_the_single_results(ctx, name, M, K):
    f = F.get(name)
    w = weights(f, M, K)
    x = torch.from_numpy(synth.make_activations(8, K, seed=3)).cuda()
    xq = ctx.quantize_q8k(x)
    one = torch.cat([ctx.gemv(f, w, xq[c:c + 1], K) for c in range(8)])
    for nb in range(2, 9):
        assert same(ctx.gemv(f, w, xq[:nb], K), one[:nb]), (name, M, K, nb)
    wide = torch.full((3, M + 5), 2.0, device="cuda")
    ctx.gemv(f, w, xq[:3], K, out=wide[:, :M], accumulate=True)
    assert same(wide[:, :M], 2.0 + one[:3]) and bool((wide[:, M:] == 2.0).all())
    ctx.check()


@pytest.mark.parametrize("name", list(F.ALL_FORMATS))
@pytest.mark.parametrize("M,K", SHAPES)
def test_act_q8_columns_are_the_single_results(ctx, name, M, K):
    f = F.get(name)
    w = weights(f, M, K)
    x = torch.from_numpy(synth.make_activations(8, K, seed=4)).cuda()
    q, d, _ = ctx.quantize_act_q8(x)
    one = torch.cat([ctx.gemv_act_q8(f, w, q[c:c + 1], d[c:c + 1], K) for c in range(8)])
    for nb in range(2, 9):
        assert same(ctx.gemv_act_q8(f, w, q[:nb], d[:nb], K), one[:nb]), (name, M, K, nb)
    ctx.check()


@pytest.mark.parametrize("name", ONE_COLUMN)
@pytest.mark.parametrize("nb", [1, 2, 3, 4, 5, 8])
def test_pass_equals_calls(ctx, name, nb):
    f, K, M1, M2 = F.get(name), 2816, 130, 77
    w1, w2 = weights(f, M1, K), weights(f, M2, K)
    x = torch.from_numpy(synth.make_activations(nb, K, seed=5)).cuda()
    ps = Pass(ctx, max_nb=nb)
    xin, xq, y = ps.buffer_f32(K), ps.buffer_q8k(K), ps.buffer_f32(M1 + M2)
    ps.quantize(xin, 0, K, xq)
    ps.gemv(ps.matrix_device(f, w1, K), xq, y, 0)
    ps.gemv(ps.matrix_device(f, w2, K), xq, y, M1)
    ps.buffer_tensor(xin).copy_(x)
    ps.run(nb)
    torch.cuda.synchronize()
    ctx.check()
    got = ps.buffer_tensor(y).clone()
    ps.close()
    xq8 = ctx.quantize_q8k(x)
    assert same(got[:, :M1], ctx.gemv(f, w1, xq8, K)) and same(got[:, M1:], ctx.gemv(f, w2, xq8, K))
