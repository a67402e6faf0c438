"""Both sides of the line between operand A in tensor memory and in shared memory, with the cut forced (the own rule cuts so small a
matrix into small tiles): one tile of 241 and of 256 tokens (the widest accumulator beside operand A), one of 257 and more, alone,
with K shared (operand A in shared memory) and without (pairs of CTAs, unless there is one row tile).  Rows that start on an even
address only, outputs that are added to, guard columns; bounds as for the other cuts, against the same rounded weights."""
import pytest
import torch

from qwengine_b200 import formats as F
from test_gpu_prefill_cuts import check

pytestmark = pytest.mark.gpu

TMEM = [(129, 512, 241, 1, 1, 6, 2), (257, 1024, 256, 1, 1, 2, 6), (128, 256, 256, 1, 1, 0, 0), (131, 768, 255, 1, 2, 16, 0), (130, 1280, 500, 2, 1, 0, 14)]
SMEM = [(130, 1280, 257, 1, 2, 6, 2), (131, 768, 512, 1, 3, 0, 0), (100, 512, 300, 1, 1, 2, 2), (257, 2304, 1000, 2, 4, 16, 16)]
PAIR = [(129, 512, 257, 1, 1, 6, 2), (257, 512, 512, 1, 1, 0, 2), (383, 1280, 300, 1, 1, 16, 0), (256, 768, 1025, 3, 1, 2, 14), (130, 1024, 545, 2, 1, 0, 0)]


@pytest.mark.parametrize("name", sorted(F.ALL_FORMATS))
@pytest.mark.parametrize("M,K,B,tiles,splits,pad,shift", TMEM + SMEM + PAIR)
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_operand_modes(ctx, name, M, K, B, tiles, splits, pad, shift, dt):
    check(ctx, name, M, K, B, dt, tiles, splits, pad, shift, accumulate=(M + B) % 2 == 1)
