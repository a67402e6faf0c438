"""The several-column kernel where its plan changes: rows whose super-blocks do not divide among the warps, one super-block more
or less than the warps, rows cut into K-parts and the longest ones, padded rows; columns that the quantizer folded into the
kernel forms from floats of every size class.  Against the oracle: exact integer sums, so within float rounding of the sum of
|w x|: 2^-23 for the products plus one rounding per partial sum, 2e-6 as in the other tests."""
import numpy as np
import pytest
import torch

import oracle
from qwengine_b200 import Pass, formats as F, synth

pytestmark = pytest.mark.gpu
EDGES = [256, 512, 4864, 5120, 5376, 8192, 8448, 10240, 30720]   # 1, 2, 19, 20, 21, 32, 33 (two parts), 40, 120 super-blocks


def within(f, w, xq, y, K):
    for c in range(xq.shape[0]):
        ref, mag = oracle.port.row_ref_mag(f.type_id, w, xq[c], K)
        assert np.max(np.abs(y[c] - ref) / mag) < 2e-6, (f.name, K, c)


@pytest.mark.parametrize("name", sorted(F.ALL_FORMATS))
@pytest.mark.parametrize("K", EDGES)
def test_row_lengths(ctx, name, K):
    f, M = F.get(name), 37
    rb = f.row_bytes(K) + 16
    w = np.zeros((M, rb), np.uint8)
    w[:, :rb - 16] = synth.make_weights(f, M, K, seed=K, scale=2e-4 if name == "IQ3_XXS" else 1e-3)
    wd = torch.from_numpy(w).cuda()
    packed = torch.from_numpy(np.ascontiguousarray(w[:, :rb - 16])).cuda()
    xq = oracle.port.quantize_q8k(synth.make_activations(8, K, seed=K + 1))
    xd = torch.from_numpy(xq).cuda()
    wide = ctx.gemv(f, wd, xd, K)
    within(f, w[:, :rb - 16], xq, wide.cpu().numpy(), K)
    for nb in (2, 5):
        for m in (wd, packed):
            got = ctx.gemv(f, m, xd[:nb], K)
            assert torch.equal(got.view(torch.int32), wide[:nb].view(torch.int32)), (name, K, nb)
    ctx.check()


@pytest.mark.parametrize("name", ["Q4_K", "IQ4_XS", "Q2_K", "IQ2_XS"])
@pytest.mark.parametrize("K", [512, 5376, 8448])
def test_columns_formed_in_the_kernel(ctx, name, K):
    """A recorded pass folds the quantizer into the matvec: the blocks are the quantizer's for zeros, values whose scale
    or its reciprocal leaves the range of the fast rounding, ties of +m and -m, infinities and NaN."""
    f, M, nb = F.get(name), 33, 6
    w = torch.from_numpy(synth.make_weights(f, M, K, seed=3, scale=1e-3)).cuda()
    x = synth.make_activations(nb, K, seed=4)
    x[1] = 0.0
    x[2, :256] *= 1e-33
    x[2, 256:] *= 1e30
    x[3, 5], x[3, 9] = -50.0, 50.0
    x[3, 256 + 200], x[3, 256 + 17] = -60.0, 60.0
    x[4, 40] = np.inf
    x[5, 300] = np.nan
    ps = Pass(ctx, max_nb=nb)
    xin, xq, y = ps.buffer_f32(K), ps.buffer_q8k(K), ps.buffer_f32(M)
    ps.quantize(xin, 0, K, xq)
    ps.gemv(ps.matrix_device(f, w, K), xq, y, 0)
    ps.buffer_tensor(xin).copy_(torch.from_numpy(x))
    ps.run(nb)
    torch.cuda.synchronize()
    ctx.check()
    got = ps.buffer_tensor(y).clone()
    ps.close()
    want = ctx.gemv(f, w, ctx.quantize_q8k(torch.from_numpy(x).cuda()), K)
    same = (got.view(torch.int32) == want.view(torch.int32)) | (got.isnan() & want.isnan())
    assert bool(same.all())
