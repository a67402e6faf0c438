"""GPU-free check of the fragment builders as the several-column kernel runs them on Q8_K columns (all thirteen formats): sign
masks and minima from the staged tables, grids as eight-byte entries, zero halves (tests/host_emul/emul_staged.cpp), a 16-row
tile against the oracle.  The integer sums are exact, so only the float additions of K / 256 super-blocks (Q8_0: K / 32 blocks)
differ: 2^-23 of sum |w x| each, 32 of them below 4e-6, and 1e-6 for the four or five of the others, as in test_decode_emul.py."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import oracle
from qwengine_b200 import formats as F, synth

HERE = os.path.dirname(os.path.abspath(__file__))
ALIGN = {"Q4_K": 16, "Q5_K": 16, "IQ4_XS": 8, "Q2_K": 4}


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("emul") / "libemul_staged.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-o", so, os.path.join(HERE, "host_emul", "emul_staged.cpp"), "-lpthread"], check=True)
    lib = C.CDLL(so)
    u8p = np.ctypeslib.ndpointer(np.uint8, flags="C_CONTIGUOUS")
    lib.emul_staged_tile.argtypes = [C.c_int, C.c_int, u8p, u8p, C.c_int, C.c_int, np.ctypeslib.ndpointer(np.float32, flags="C_CONTIGUOUS")]
    return lib


@pytest.mark.parametrize("name", sorted(F.ALL_FORMATS))
@pytest.mark.parametrize("nb,addr_lo", [(2, 0), (7, 8), (8, 2)])
@pytest.mark.parametrize("extreme", [False, True])
def test_tile_matches_oracle(emul, name, nb, addr_lo, extreme):
    f, K = F.get(name), 1024
    w = synth.make_weights(f, 16, K, seed=5, scale=2e-4 if name == "IQ3_XXS" else 1e-3)
    x = synth.make_activations(nb, K, seed=6) * (np.arange(nb, dtype=np.float32)[:, None] + 1)
    if extreme:      # the largest sums of a sub-block, both signs: both ends of the two digits
        x = np.where(np.arange(K) // 64 % 2 == 0, 127.0, -127.0).astype(np.float32) * np.ones((nb, 1), np.float32)
    xq = oracle.port.quantize_q8k(x)
    y = np.zeros((16, 8), np.float32)
    assert emul.emul_staged_tile(f.type_id, K, w.reshape(-1), xq.reshape(-1), nb, addr_lo if addr_lo % ALIGN.get(name, 2) == 0 else 0, y) == 0
    for c in range(nb):
        ref, mag = oracle.port.row_ref_mag(f.type_id, w, xq[c], K)
        assert np.max(np.abs(y[:, c] - ref) / mag) < (4e-6 if name == "Q8_0" else 1e-6)
