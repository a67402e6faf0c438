"""The prefill GEMM at the edges of its cuts: token tiles of one or two accumulators whose last one is ragged, a tile's K
shared by up to eight CTAs (more than it has super-blocks divide evenly into), strided rows that start at even addresses,
a matrix that starts and ends inside a 16-byte unit.  Against torch on the weights of q38b_dequant_rows rounded to the
operand type, fp32 accumulation: the same operands for all but Q4_K, Q5_K, Q6_K, so that only the order of the additions
differs (1e-5 of sum |w x|, the bound of the other prefill tests); those three round scale and minimum first (2^-8 of a
weight in bf16, 2^-10 in fp16)."""
import pytest
import torch

from qwengine_b200 import api, formats as F, synth

pytestmark = pytest.mark.gpu
PACKED = ("Q4_K", "Q5_K", "Q6_K")


def check(ctx, name, M, K, B, dt, tiles, splits, pad=0, shift=0, accumulate=False):
    f = F.get(name)
    rb = f.row_bytes(K) + pad
    buf = torch.full((M * rb + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    w = buf[shift:shift + M * rb].view(M, rb)
    w[:, :f.row_bytes(K)].copy_(torch.from_numpy(synth.make_weights(f, M, K, seed=M + K)))
    x = torch.randn((B, K), device="cuda", generator=torch.Generator("cuda").manual_seed(B)).to(dt)
    ldy = M + 3
    y = torch.full((B, ldy), 7.0, device="cuda")
    fn = ctx.lib.q38b_gemm_prefill if dt == torch.bfloat16 else ctx.lib.q38b_gemm_prefill_f16
    st = torch.cuda.current_stream().cuda_stream
    assert ctx.lib.q38b_debug_set_prefill_cut(ctx.h, tiles, splits) == 0
    try:
        rc = fn(ctx.h, f.type_id, w.data_ptr(), rb, K, M, x.data_ptr(), K, B, y.data_ptr(), ldy, int(accumulate), st)
    finally:
        ctx.lib.q38b_debug_set_prefill_cut(ctx.h, 0, 0)
    assert rc == 0
    ctx.check()
    wq = torch.empty((M, K), dtype=dt, device="cuda")
    assert ctx.lib.q38b_dequant_rows(ctx.h, f.type_id, w.data_ptr(), rb, K, M, wq.data_ptr(), api.OUT_BF16 if dt == torch.bfloat16 else api.OUT_F16, st) == 0
    ref, mag = x.double() @ wq.double().t(), x.double().abs() @ wq.double().abs().t()
    got = y[:, :M].double() - (7.0 if accumulate else 0.0)
    err = ((got - ref).abs() - (7.0 * 2 ** -23 if accumulate else 0.0)) / mag
    packed = name == "Q6_K" or (name in PACKED and (w.data_ptr() | rb) % 4 == 0)   # rows of Q4_K, Q5_K that are 2-byte aligned only: exact
    bound = (4e-3 if dt == torch.bfloat16 else 1e-3) if packed else 1e-5
    assert float(err.max()) < bound, (name, M, K, B, tiles, splits, float(err.max()))
    assert bool((y[:, M:] == 7.0).all())


@pytest.mark.parametrize("name", list(F.ALL_FORMATS))
@pytest.mark.parametrize("M,K,B,pad,shift,tiles,splits", [
    (130, 768, 17, 0, 0, 1, 1), (129, 1280, 40, 6, 2, 1, 3), (64, 2048, 300, 0, 0, 1, 2), (257, 2304, 520, 16, 16, 2, 4), (128, 256, 1, 2, 14, 1, 1)])
def test_cuts_all_formats(ctx, name, M, K, B, pad, shift, tiles, splits):
    check(ctx, name, M, K, B, torch.bfloat16 if B != 40 else torch.float16, tiles, splits, pad, shift)


@pytest.mark.parametrize("splits", [1, 2, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("B,tiles", [(16, 1), (77, 1), (250, 1), (250, 3), (258, 1), (530, 2)])
def test_splits_and_tiles(ctx, splits, B, tiles):
    check(ctx, "IQ3_XXS", 200, 2304, B, torch.bfloat16, tiles, splits, accumulate=splits % 2 == 0)
    check(ctx, "Q5_K", 200, 2304, B, torch.float16, tiles, splits, accumulate=splits % 2 == 1)


@pytest.mark.parametrize("name", ["IQ3_XXS", "Q5_K"])
def test_full_tiles_fill_the_exchange(ctx, name):
    """Two accumulators of 256 tokens: the partial sums of three other CTAs take the rings to the last byte, a fourth's have
    no room (refused: the own rule never picks that cut)."""
    for splits in (2, 3, 4):
        check(ctx, name, 130, 2304, 512, torch.bfloat16, 1, splits)
    f, K = F.get(name), 2304
    w = torch.zeros((130, f.row_bytes(K)), dtype=torch.uint8, device="cuda")
    x = torch.zeros((512, K), dtype=torch.bfloat16, device="cuda")
    assert ctx.lib.q38b_debug_set_prefill_cut(ctx.h, 1, 5) == 0
    try:
        with pytest.raises(api.Q38BError) as e:
            ctx.gemm_prefill(f, w, x, K)
    finally:
        ctx.lib.q38b_debug_set_prefill_cut(ctx.h, 0, 0)
    assert e.value.status == -6      # Q38B_ERR_NOMEM


@pytest.mark.parametrize("name", ["Q4_K", "Q5_K"])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("pad,shift", [(4, 4), (0, 8), (12, 0)])
def test_packed_conversion_on_unaligned_rows(ctx, name, dt, pad, shift):
    """Rows that are 4- but not 16-byte aligned: the packed conversion behind the word loads that assume two bytes only."""
    check(ctx, name, 130, 1280, 33, dt, 1, 2, pad, shift)


@pytest.mark.parametrize("M,K,B", [(5120, 5120, 9), (640, 17408, 77), (17000, 1024, 513), (1024, 512, 1030)])
def test_own_rule(ctx, M, K, B):
    check(ctx, "Q4_K", M, K, B, torch.bfloat16, 0, 0)
    check(ctx, "IQ2_XS", M, K, B, torch.float16, 0, 0)
