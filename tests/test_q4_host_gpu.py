"""The call on host arrays: ordinary, page-locked and mixed ones, rows that fit the kept pages and rows that do not, sizes growing and
shrinking, several threads on one context; the same bits as the call on device arrays."""
import ctypes as C
import threading

import numpy as np
import pytest

from makepad_b200 import _lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(1, 32), (1000, 2112), (12288, 4096)])
def test_host_arrays_of_every_kind(orc, N, K):
    import makepad_b200
    import torch
    ctx = makepad_b200.Context(0)
    codes, scales = synth.q4_weight(N, K, seed=81)
    w = makepad_b200.Q4Weight(ctx, codes, scales)
    lin = makepad_b200.QuantLinear(w)

    def call(x, y):
        ctx.check(ctx.lib.mpq_q4_linear_forward_host(ctx.h, w.h, C.c_void_p(x.ctypes.data), x.shape[0], C.c_void_p(y.ctypes.data)))

    for M in (1, 3, 40, 2, 300, 1):                          # 40 rows and more of 4096, 300 of 2112 pass the kept pages, 300 of 32 do not
        x = synth.activations(M, K, seed=82 + M)
        want = lin(torch.from_numpy(x).cuda()).cpu().numpy()
        assert np.array_equal(lin(x), want)
        locked = torch.from_numpy(x).pin_memory().numpy()
        for xs, ys in ((x, np.empty_like(want)), (locked, np.empty_like(want)), (x, torch.empty(M, N).pin_memory().numpy()),
                       (locked, torch.empty(M, N).pin_memory().numpy())):
            call(xs, ys)
            assert np.array_equal(ys, want)
    x = [synth.activations(1, K, seed=90 + i) for i in range(4)]
    want = [lin(torch.from_numpy(v).cuda()).cpu().numpy() for v in x]
    good = [True] * 4

    def work(i):
        for _ in range(50):
            good[i] &= np.array_equal(lin(x[i]), want[i])

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(good)
    w.destroy()
    assert ctx.lib.mpq_context_poll_status(ctx.h) == _lib.OK
    ctx.close()


@pytest.mark.parametrize("M,K,pages", [(1, 4096, True), (32, 4096, True), (33, 4096, False), (64, 4096, False), (23, 11008, False)])
def test_large_activations_are_copied_by_the_driver(M, K, pages):
    """Above 512 KB the copy of the activations by one host core takes longer than the driver's: no kernel that fetches them is launched."""
    import makepad_b200
    import torch
    ctx = makepad_b200.Context(0)
    codes, scales = synth.q4_weight(64, K, seed=83)
    w = makepad_b200.Q4Weight(ctx, codes, scales)
    lin = makepad_b200.QuantLinear(w)
    x = synth.activations(M, K, seed=84)
    want = lin(torch.from_numpy(x).cuda()).cpu().numpy()
    before = ctx.launches
    lin(torch.from_numpy(x).cuda())
    alone = ctx.launches - before
    before = ctx.launches
    assert np.array_equal(lin(x), want)
    assert ctx.launches - before == alone + pages
    w.destroy()
    ctx.close()
