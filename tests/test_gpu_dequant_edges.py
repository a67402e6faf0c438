"""q38b_dequant_rows where its slices, pieces and alignments can go wrong: rows of one super-block, slices of less than
four, strided rows that start at every even address, a matrix that starts inside a 16-byte unit, an output that is only
4-byte aligned, negative scales (signs of zeros).  Bit for bit against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from qwengine_b200 import api, formats as F, synth

pytestmark = pytest.mark.gpu
NP16 = {api.OUT_F16: np.float16, api.OUT_F32: np.float32}


@pytest.mark.parametrize("name", list(F.ALL_FORMATS))
@pytest.mark.parametrize("rows,K,pad,shift,out_shift", [(1, 256, 0, 0, 0), (7, 768, 6, 2, 4), (19, 1280, 2, 14, 8), (3, 1024, 0, 6, 0), (1300, 2304, 0, 0, 12)])
def test_slices_and_alignments(ctx, name, rows, K, pad, shift, out_shift):
    f = F.get(name)
    w = synth.make_weights(f, rows, K, seed=rows + K)
    if f.name in ("Q6_K", "Q8_0", "IQ4_XS"):              # a negative super-scale: zeros keep the sign the multiplication gives
        at = {"Q6_K": 209, "Q8_0": 1, "IQ4_XS": 1}[f.name]
        w.reshape(rows, -1, f.block_bytes)[:, ::2, at] |= 0x80
    want = oracle.port.dequantize(f.type_id, w)
    rb = f.row_bytes(K) + pad
    buf = torch.zeros(rows * rb + 64, dtype=torch.uint8, device="cuda")
    view = buf[shift:shift + rows * rb].view(rows, rb)
    view[:, :f.row_bytes(K)].copy_(torch.from_numpy(w))
    for kind in (api.OUT_F32, api.OUT_F16, api.OUT_BF16):
        es = 4 if kind == api.OUT_F32 else 2
        out = torch.full((rows * K * es + 64,), 0xEE, dtype=torch.uint8, device="cuda")
        rc = ctx.lib.q38b_dequant_rows(ctx.h, f.type_id, view.data_ptr(), rb, K, rows, out.data_ptr() + out_shift, kind, torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        got = out.cpu()
        assert bool((got[:out_shift] == 0xEE).all()) and bool((got[out_shift + rows * K * es:] == 0xEE).all())
        got = got[out_shift:out_shift + rows * K * es].clone()
        if kind == api.OUT_BF16:
            assert torch.equal(got.view(torch.int16).view(rows, K), torch.from_numpy(want).to(torch.bfloat16).view(torch.int16))
        else:
            exp = want.astype(NP16[kind])
            assert np.array_equal(got.numpy().view(exp.dtype).reshape(rows, K).view(np.uint8), exp.view(np.uint8))
