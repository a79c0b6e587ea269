"""The streaming kernel's runs: one, two and four chunks per copy, whole tiles per CTA with fewer groups than warps and with several tiles
shared by the same warps, equal runs cut between CTAs, one and several rows, plain and with SwiGLU in the staging."""
import os

import numpy as np
import pytest

from makepad_b200 import _lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", ["0", "1", "2", "4"])
def test_runs_of_the_streaming_kernel(orc, group):
    import makepad_b200
    import torch
    os.environ["MPQ_Q4_GROUP"] = group
    try:
        c = makepad_b200.Context(0)
    finally:
        del os.environ["MPQ_Q4_GROUP"]
    # one group in all; equal runs (few rows); whole tiles: 1, 2 and 3 groups of four chunks per CTA, about 2.6 tiles per CTA; a K for which
    # only short copies fit beside the row
    for N, K in [(1, 32), (33, 160), (100, 4096), (1000, 2112), (3000, 64), (3000, 512), (4100, 736), (12300, 1024), (2900, 28672)]:
        codes, scales = synth.q4_weight(N, K, seed=61)
        w = makepad_b200.Q4Weight(c, codes, scales)
        lin = makepad_b200.QuantLinear(w)
        for M in (1, 3):
            if M * K >= 16384 and M > 1:
                continue                                          # several rows of a long K go to another kernel
            x = synth.activations(M, K, seed=62)
            buf = torch.full((M * N + 256,), 777.0, device="cuda")
            y = buf[128:128 + M * N].view(M, N)
            lin.forward(torch.from_numpy(x).cuda(), out=y)
            torch.cuda.synchronize()
            rep = orc.err_report(y.cpu().numpy(), orc.q4_matmul_f64(codes, scales, x))
            # as for every Q4 output: products exact to 22 bits, fp32 sums
            assert rep["floored_1e-2_rms"] < 1e-3 and rep["max_abs_over_rms"] < 2e-5, (N, K, M, rep)
            assert (buf[:128] == 777.0).all() and (buf[128 + M * N:] == 777.0).all()
            gate_up = torch.from_numpy(synth.activations(M, 2 * K, seed=63)).cuda()
            assert torch.equal(lin.forward_swiglu(gate_up), lin(makepad_b200.swiglu(c, gate_up))), (N, K, M)
        w.destroy()
    assert c.lib.mpq_context_poll_status(c.h) == _lib.OK
    c.close()


@pytest.mark.parametrize("tile", ["1", "0"])
@pytest.mark.parametrize("N,K", [(28456, 320), (28300, 1088), (50000, 128), (24000, 768)])
def test_many_tiles_per_cta(orc, monkeypatch, N, K, tile):
    """More than four tiles of a CTA are shared between its warps (fewer take another way through the merge); with equal runs (tile 0) its
    first and last tile are shared with the neighbours as well."""
    import makepad_b200
    import torch
    monkeypatch.setenv("MPQ_Q4_TILE", tile)
    c = makepad_b200.Context(0)
    codes, scales = synth.q4_weight(N, K, seed=64)
    w = makepad_b200.Q4Weight(c, codes, scales)
    lin = makepad_b200.QuantLinear(w)
    for M in (1, 2, 4):
        x = synth.activations(M, K, seed=65)
        xd = torch.from_numpy(x).cuda()
        buf = torch.full((M * N + 256,), 777.0, device="cuda")
        y = buf[128:128 + M * N].view(M, N)
        lin.forward(xd, out=y)
        assert torch.equal(y, lin(xd))
        rep = orc.err_report(y.cpu().numpy(), orc.q4_matmul_f64(codes, scales, x))
        assert rep["floored_1e-2_rms"] < 1e-3 and rep["max_abs_over_rms"] < 2e-5, (N, K, M, rep)
        assert (buf[:128] == 777.0).all() and (buf[128 + M * N:] == 777.0).all()
    w.destroy()
    assert c.lib.mpq_context_poll_status(c.h) == _lib.OK
    c.close()
