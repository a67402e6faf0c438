"""Two to four columns on the one-column kernel's granules (q38b_gemv1.cuh, NC = 2 and 4): every format, Q8_K blocks and per-32
columns, rows whose super-blocks do not fill a slice or fall short of the warps, ragged tiles, padded rows, strided outputs that are
added to, several matrices of a recorded pass with the columns given as floats.  Each column must be the single column's result and
the several-column kernel's, bit for bit: the same integer sums, float products and order."""
import pytest
import torch

from qwengine_b200 import Pass, formats as F, synth

pytestmark = pytest.mark.gpu
ONE_COLUMN_BITS = ("Q2_K", "IQ2_XXS", "IQ2_XS", "IQ2_S", "IQ1_S", "IQ1_M")


@pytest.fixture
def route(ctx):
    yield lambda mode: ctx.lib.q38b_debug_set_cols_route(ctx.h, mode)
    ctx.lib.q38b_debug_set_cols_route(ctx.h, 0)
    ctx.debug_set_rowgroup(True)


def bits(t):
    return t.contiguous().view(torch.int32)


@pytest.mark.parametrize("name", sorted(F.ALL_FORMATS))
@pytest.mark.parametrize("M,K,pad", [(1, 256, 0), (37, 1280, 16), (83, 4864, 0), (2403, 2816, 0), (40, 8448, 0), (19, 17408, 32)])
def test_columns_are_the_single_columns(ctx, route, name, M, K, pad):
    f = F.get(name)
    rb = f.row_bytes(K) + pad
    w = torch.zeros((M, rb), dtype=torch.uint8, device="cuda")
    w[:, :rb - pad].copy_(torch.from_numpy(synth.make_weights(f, M, K, seed=K + M)))
    x = torch.from_numpy(synth.make_activations(4, K, seed=M)).cuda()
    x[1, :300] = 0.0
    q8, (q, d, _) = ctx.quantize_q8k(x), ctx.quantize_act_q8(x)
    ctx.debug_set_rowgroup(False)
    one = torch.cat([ctx.gemv(f, w, q8[c:c + 1], K) for c in range(4)])
    one32 = torch.cat([ctx.gemv_act_q8(f, w, q[c:c + 1], d[c:c + 1], K) for c in range(4)])
    parts = K > 8192 and name not in ONE_COLUMN_BITS
    for mode in (2, 1, 0):
        route(mode)
        for nb in (2, 3, 4):
            y = torch.full((nb, M + 5), 3.0, device="cuda")
            got = ctx.gemv_act_q8(f, w, q[:nb], d[:nb], K, out=y[:, :M])
            assert torch.equal(bits(got), bits(one32[:nb])), (mode, nb)
            ctx.gemv_act_q8(f, w, q[:nb], d[:nb], K, out=y[:, :M], accumulate=True)
            assert torch.equal(bits(y[:, :M]), bits(one32[:nb] + one32[:nb])) and bool((y[:, M:] == 3.0).all())
            if not parts:
                y = torch.full((nb, M + 5), 3.0, device="cuda")
                ctx.gemv(f, w, q8[:nb], K, out=y[:, :M])
                assert torch.equal(bits(y[:, :M]), bits(one[:nb])) and bool((y[:, M:] == 3.0).all()), (mode, nb)
    ctx.check()


@pytest.mark.parametrize("name", sorted(F.ALL_FORMATS))
@pytest.mark.parametrize("nb", [2, 3, 4])
def test_columns_of_a_pass(ctx, route, name, nb):
    """Two matrices on columns that the kernel forms from floats, among them zeros, infinities and NaN."""
    f, K, Ms = F.get(name), 2816, (67, 24)
    x = torch.from_numpy(synth.make_activations(nb, K, seed=nb)).cuda()
    x[0, 256:512] = 0.0
    x[1, 7], x[nb - 1, 700] = float("inf"), float("nan")
    ws = [torch.from_numpy(synth.make_weights(f, M, K, seed=M)).cuda() for M in Ms]
    outs = []
    for mode in (2, 1):
        route(mode)
        ps = Pass(ctx, max_nb=nb)
        xin, xq, y = ps.buffer_f32(K), ps.buffer_q8k(K), ps.buffer_f32(sum(Ms))
        ps.quantize(xin, 0, K, xq)
        for i, w in enumerate(ws):
            ps.gemv(ps.matrix_device(f, w, K), xq, y, i * Ms[0])
        ps.buffer_tensor(xin).copy_(x)
        ps.run(nb)
        torch.cuda.synchronize()
        ctx.check()
        outs.append(ps.buffer_tensor(y).clone())
        ps.close()
    same = (bits(outs[0]) == bits(outs[1])) | (outs[0].isnan() & outs[1].isnan())
    assert bool(same.all())
