"""The kernels that add the partial outputs of a Q4 call (K slices up to 16 rows, pieces of a batch above): few and many of them, rows
that float4 accesses fit and rows that they do not, columns up to the edge of the output and none behind it."""
import numpy as np
import pytest

from makepad_b200 import _lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(257, 11008), (260, 11008), (513, 28672), (516, 1024)])
def test_partial_outputs_are_added(ctx, orc, N, K):
    import makepad_b200
    import torch
    codes, scales = synth.q4_weight(N, K, seed=51)
    w = makepad_b200.Q4Weight(ctx, codes, scales)
    lin = makepad_b200.QuantLinear(w)
    for M in (5, 16, 17, 33, 64):
        x = synth.activations(M, K, seed=52 + M)
        buf = torch.full((M * N + 256,), 777.0, device="cuda")
        y = buf[128:128 + M * N].view(M, N)
        lin.forward(torch.from_numpy(x).cuda(), out=y)
        torch.cuda.synchronize()
        rep = orc.err_report(y.cpu().numpy(), orc.q4_matmul_f64(codes, scales, x))
        # as for every Q4 output: products exact to 22 bits, fp32 sums
        assert rep["floored_1e-2_rms"] < 1e-3 and rep["max_abs_over_rms"] < 2e-5, (N, K, M, rep)
        assert (buf[:128] == 777.0).all() and (buf[128 + M * N:] == 777.0).all()
    w.destroy()
    assert ctx.lib.mpq_context_poll_status(ctx.h) == _lib.OK
