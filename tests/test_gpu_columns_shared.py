"""Launches that several columns or several outputs share: the copies of the outputs that a sharded run's peers keep (here
buffers of this device), and calls that overlap on two streams."""
import ctypes as C

import pytest
import torch

from qwengine_b200 import api, formats as F, synth

pytestmark = pytest.mark.gpu
ONE_COLUMN = ["Q2_K", "IQ2_XXS", "IQ2_XS", "IQ2_S", "IQ1_S", "IQ1_M"]


def weights(f, M, K):
    return torch.from_numpy(synth.make_weights(f, M, K, seed=M + K)).cuda()


def same(a, b):
    return torch.equal(a.contiguous().view(torch.int32), b.contiguous().view(torch.int32))


def pointers(ts):
    return (C.c_void_p * len(ts))(*[t.data_ptr() for t in ts])


@pytest.mark.parametrize("name", ONE_COLUMN + ["Q4_K"])
@pytest.mark.parametrize("nb", [2, 3, 4])
@pytest.mark.parametrize("floats", [False, True])
def test_merged_launch_stores_the_peers_copies(ctx, name, nb, floats):
    f, K, Ms, n_peers = F.get(name), 1280, (130, 77), 2
    ws = [weights(f, M, K) for M in Ms]
    x = torch.from_numpy(synth.make_activations(nb, K, seed=7)).cuda()
    xq = ctx.quantize_q8k(x)
    outs = [[torch.full((nb, M + 3 + i), 9.0, device="cuda") for _ in range(1 + n_peers)] for i, M in enumerate(Ms)]
    fn = ctx.lib.q38b_gemvn_group_x
    fn.argtypes = [C.c_void_p, C.c_uint32, C.c_int, C.c_void_p, C.c_size_t, C.c_int, C.c_void_p, C.c_void_p, C.c_longlong, C.c_void_p,
                   C.c_longlong, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]
    lds = (C.c_longlong * 2)(*[o[0].stride(0) for o in outs])
    rc = fn(ctx.h, f.type_id, 2, pointers(ws), f.row_bytes(K), K, (C.c_int * 2)(*Ms), None if floats else xq.data_ptr(), 0 if floats else K // 256,
            x.data_ptr() if floats else None, K if floats else 0, nb, pointers([o[0] for o in outs]), lds,
            pointers([o[1 + p] for o in outs for p in range(n_peers)]), n_peers, api._stream())
    assert rc == 0
    ctx.check()
    for M, w, o in zip(Ms, ws, outs):
        want = ctx.gemv(f, w, xq, K)
        for t in o:
            assert same(t[:, :M], want) and bool((t[:, M:] == 9.0).all())


@pytest.mark.parametrize("name", ONE_COLUMN)
@pytest.mark.parametrize("nb", [1, 4, 5, 8])
def test_scatter_stores_the_peers_copies(ctx, name, nb):
    f, K, M = F.get(name), 2816, 131
    w = weights(f, M, K)
    xq = ctx.quantize_q8k(torch.from_numpy(synth.make_activations(nb, K, seed=8)).cuda())
    outs = [torch.full((nb, M + 5), 9.0, device="cuda") for _ in range(3)]
    fn = ctx.lib.q38b_gemv_q8k_scatter
    fn.argtypes = [C.c_void_p, C.c_uint32, C.c_void_p, C.c_size_t, C.c_int, C.c_int, C.c_void_p, C.c_longlong, C.c_int, C.c_void_p, C.c_longlong,
                   C.c_int, C.c_void_p, C.c_int, C.c_void_p]
    assert fn(ctx.h, f.type_id, w.data_ptr(), f.row_bytes(K), K, M, xq.data_ptr(), K // 256, nb, outs[0].data_ptr(), M + 5, 0, pointers(outs[1:]), 2,
              api._stream()) == 0
    ctx.check()
    want = ctx.gemv(f, w, xq, K)
    for t in outs:
        assert same(t[:, :M], want) and bool((t[:, M:] == 9.0).all())


def test_calls_on_two_streams(ctx):
    """Matvecs of several columns, GEMMs whose tiles share K in clusters and dense dequantization keep nothing between
    calls: two streams that run them at the same time get the results of one after the other."""
    K, M = 5120, 3001
    jobs = []
    for i, name in enumerate(["IQ2_XS", "IQ3_XXS", "IQ1_M", "Q4_K"]):
        f = F.get(name)
        w = weights(f, M, K)
        x = torch.from_numpy(synth.make_activations(4, K, seed=20 + i)).cuda()
        xb = torch.randn((77, K), device="cuda", generator=torch.Generator("cuda").manual_seed(i)).to(torch.bfloat16)
        xq = ctx.quantize_q8k(x) if name.startswith(("IQ2", "IQ1")) else None
        q, d, _ = ctx.quantize_act_q8(x)

        def job(f=f, w=w, xq=xq, q=q, d=d, xb=xb):
            out = [ctx.gemv_act_q8(f, w, q, d, K), ctx.gemm_prefill(f, w, xb, K), ctx.dequant_rows(f, w, K)]
            return out + ([ctx.gemv(f, w, xq, K)] if xq is not None else [])
        jobs.append(job)
    want = [job() for job in jobs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = {}
    for _ in range(3):
        for i, job in enumerate(jobs):
            with torch.cuda.stream(streams[i % 2]):
                got[i] = job()
    torch.cuda.synchronize()
    ctx.check()
    for i, w in enumerate(want):
        assert all(same(a, b) for a, b in zip(got[i], w)), i
