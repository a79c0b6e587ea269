"""The GEMM of few activation rows (weights as the M operand): both atoms of a weight tile, the last tile with one, rows up to the edges of
the operand's steps of 16, K that fills its blocks and not, K whole and cut; nothing outside the output, the same bits twice and under capture."""
import os

import numpy as np
import pytest

from makepad_b200 import _lib, synth

pytestmark = pytest.mark.gpu


def _bits(y):
    import torch
    return y.view(torch.int16).cpu().numpy().view(np.uint16)


@pytest.mark.parametrize("splits", ["0", "1", "3", "16"])
@pytest.mark.parametrize("N,K", [(8, 32), (128, 256), (136, 1056), (224, 288), (352, 4096), (360, 6176), (4096, 2048)])
def test_few_rows_against_the_oracle(ctx, orc, monkeypatch, N, K, splits):
    import makepad_b200
    import torch
    if splits != "0":
        monkeypatch.setenv("MPQ_FP4_KERNEL", "rows=" + splits)
    b, sfb = synth.nvfp4_tensor(N, K, seed=91, stream=1)
    lin = makepad_b200.QuantLinear(makepad_b200.Nvfp4Weight(ctx, b, sfb, 2.0))
    for M in (1, 15, 16, 17, 33, 48, 64):
        a, sfa = synth.nvfp4_tensor(M, K, seed=92 + M, stream=0)
        ad, sd = torch.from_numpy(a).cuda(), torch.from_numpy(sfa).cuda()
        buf = torch.full((M * N + 128,), 7.0, dtype=torch.bfloat16, device="cuda")
        y = buf[64:64 + M * N].view(M, N)
        lin.forward((ad, sd, 0.5), out=y)
        assert torch.equal(y, lin((ad, sd, 0.5)))
        torch.cuda.synchronize()
        assert ctx.lib.mpq_context_poll_status(ctx.h) == _lib.OK
        assert (buf[:64] == 7.0).all() and (buf[64 + M * N:] == 7.0).all()
        c32, c16 = orc.nvfp4_gemm(a, sfa, 0.5, b, sfb, 2.0)
        got = orc.bf16_bits_to_f32(_bits(y))
        # fp32 sums of exact products, rounded once to bf16: within one bf16 ulp of the binary32 oracle, and mostly the same bits
        assert np.all(np.abs(got - c32) <= np.maximum(2.0 ** -7 * np.abs(c32), 1e-5 * np.sqrt(np.mean(c32 * c32)))), (M, N, K)
        assert np.mean(_bits(y) == c16) > 0.98, (M, N, K)
        if M == 17:
            graph, z = torch.cuda.CUDAGraph(), torch.empty_like(y)
            with torch.cuda.graph(graph):
                lin.forward((ad, sd, 0.5), out=z)
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(z, y)
            del graph


def test_a_loaded_weight_takes_few_rows(ctx, tmp_path):
    """The maps of a weight are made again when it is read from its file."""
    import makepad_b200
    import torch
    b, sfb = synth.nvfp4_tensor(456, 512, seed=95, stream=1)
    w = makepad_b200.Nvfp4Weight(ctx, b, sfb, 1.0)
    path = os.path.join(tmp_path, "w.mpq")
    w.save(path)
    a, sfa = (torch.from_numpy(v).cuda() for v in synth.nvfp4_tensor(5, 512, seed=96, stream=0))
    w2 = makepad_b200.load_weight(ctx, path)
    assert torch.equal(makepad_b200.QuantLinear(w)((a, sfa, 1.0)), makepad_b200.QuantLinear(w2)((a, sfa, 1.0)))


@pytest.mark.parametrize("M", [16, 1000])
def test_an_uncut_call_reserves_the_room_of_later_captures(M):
    """The context's first call is one of few rows whose K is not cut; a captured call of few rows or of many, whose K is, then has the two
    launches and the bits of the eager one."""
    import makepad_b200
    import torch
    N, K = 4096, 14336
    c2 = makepad_b200.Context(0)
    small = makepad_b200.QuantLinear(makepad_b200.Nvfp4Weight(c2, *synth.nvfp4_tensor(8, 32, seed=97, stream=1), 1.0))
    lin = makepad_b200.QuantLinear(makepad_b200.Nvfp4Weight(c2, *synth.nvfp4_tensor(N, K, seed=98, stream=1), 1.0))
    rows = lambda m, k: (*(torch.from_numpy(v).cuda() for v in synth.nvfp4_tensor(m, k, seed=99, stream=0)), 0.5)
    a, y = rows(M, K), torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    before = c2.launches
    small(rows(5, 32))
    torch.cuda.synchronize()
    assert c2.launches - before == 1
    graph = torch.cuda.CUDAGraph()
    before = c2.launches
    with torch.cuda.graph(graph):
        lin.forward(a, out=y)
    assert c2.launches - before == 2
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, lin(a))
    assert c2.lib.mpq_context_poll_status(c2.h) == _lib.OK
    del graph
    c2.close()
