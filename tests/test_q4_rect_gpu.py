"""The rectangle kernel's K slices: one, several that a cluster adds, several that go through memory; few groups per CTA, tiles shared by
warps and not, the last slice shorter, every MMA tile count; the three forms agree to rounding and each gives the same bits twice."""
import os

import numpy as np
import pytest

from makepad_b200 import _lib, synth

pytestmark = pytest.mark.gpu


def _context(**env):
    import makepad_b200
    os.environ.update(env)
    try:
        return makepad_b200.Context(0)
    finally:
        for k in env:
            del os.environ[k]


@pytest.mark.parametrize("N,K", [(1, 256), (33, 1120), (257, 4096), (1000, 2112), (4096, 11008), (12300, 1024), (300, 28672)])
def test_slices_of_the_rectangle_kernel(orc, N, K):
    import makepad_b200
    import torch
    codes, scales = synth.q4_weight(N, K, seed=71)
    contexts = [_context(MPQ_Q4_STREAM="0", MPQ_Q4_RECT_CLUSTER=c, MPQ_Q4_RECT_NKS=n) for c in "01" for n in ("0", "2", "3", "5", "8")]
    for M in (2, 5, 12, 16):
        x = synth.activations(M, K, seed=72)
        xd = torch.from_numpy(x).cuda()
        ref = orc.q4_matmul_f64(codes, scales, x)
        for c in contexts:
            w = makepad_b200.Q4Weight(c, codes, scales)
            lin = makepad_b200.QuantLinear(w)
            buf = torch.full((M * N + 256,), 777.0, device="cuda")
            y = buf[128:128 + M * N].view(M, N)
            lin.forward(xd, out=y)
            again = lin(xd)
            torch.cuda.synchronize()
            rep = orc.err_report(y.cpu().numpy(), ref)
            # as for every Q4 output: products exact to 22 bits, fp32 sums
            assert rep["floored_1e-2_rms"] < 1e-3 and rep["max_abs_over_rms"] < 2e-5, (N, K, M, rep)
            assert torch.equal(y, again)
            assert (buf[:128] == 777.0).all() and (buf[128 + M * N:] == 777.0).all()
            w.destroy()
    for c in contexts:
        assert c.lib.mpq_context_poll_status(c.h) == _lib.OK
        c.close()


# (28672 of K at 16 rows: more slices than a cluster holds)
@pytest.mark.parametrize("N,K,M,slices,one", [(4096, 4096, 8, 0, 1), (4096, 4096, 8, 5, 1), (1000, 2112, 13, 3, 1), (33, 1120, 5, 2, 1), (300, 28672, 16, 0, 2)])
def test_slices_are_added_by_a_cluster_or_by_a_second_launch(N, K, M, slices, one):
    """One launch where the slices of a tile group are a cluster (nothing but the plan says that they are), two through memory."""
    import makepad_b200
    import torch
    codes, scales = synth.q4_weight(N, K, seed=75)
    xd = torch.from_numpy(synth.activations(M, K, seed=76)).cuda()
    for cluster, launches in (("1", one), ("0", 2)):
        c = _context(MPQ_Q4_RECT_CLUSTER=cluster, MPQ_Q4_RECT_NKS=str(slices))
        w = makepad_b200.Q4Weight(c, codes, scales)
        before = c.launches
        makepad_b200.QuantLinear(w)(xd)
        assert c.launches - before == launches, (cluster, slices)
        w.destroy()
        c.close()


def test_slices_in_a_graph_and_on_two_streams(ctx, orc):
    """Clusters under capture, and calls of two contexts in flight on two streams (the calls of one context are ordered)."""
    import makepad_b200
    import torch
    N, K, M = 4096, 4096, 8
    codes, scales = synth.q4_weight(N, K, seed=73)
    contexts = [makepad_b200.Context(0) for _ in range(2)]
    lins = [makepad_b200.QuantLinear(makepad_b200.Q4Weight(c, codes, scales)) for c in contexts]
    xs = [torch.from_numpy(synth.activations(M, K, seed=74 + i)).cuda() for i in range(2)]
    want = [lin(x) for lin, x in zip(lins, xs)]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    out = torch.empty_like(want[0])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        lins[0].forward(xs[0], out=out)
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want[0])
    outs = [[torch.empty_like(want[0]) for _ in range(8)] for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    for k in range(8):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                lins[i].forward(xs[i], out=outs[i][k])
    torch.cuda.synchronize()
    assert all(torch.equal(o, want[i]) for i in range(2) for o in outs[i])
    del g
    for lin, c in zip(lins, contexts):
        assert c.lib.mpq_context_poll_status(c.h) == _lib.OK
        lin.w.destroy()
        c.close()
