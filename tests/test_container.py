"""The weight container: canonical files round-trip on the CPU; device-layout files round-trip on the GPU
without a repack pass and are refused when damaged or written for another layout."""
import ctypes as C
import os
import struct

import numpy as np
import pytest

from makepad_b200 import _lib, synth


def test_canonical_roundtrip_needs_no_gpu(tmp_path):
    import makepad_b200
    codes, scales = synth.q4_weight(96, 256, seed=1)
    p = str(tmp_path / "w.q4c")
    makepad_b200.save_canonical(p, _lib.FMT_Q4, codes, scales)
    fmt, c2, s2, ts = makepad_b200.load_canonical(p)
    assert fmt == _lib.FMT_Q4 and np.array_equal(c2, codes) and np.array_equal(s2, scales) and ts == 1.0
    b, sfb = synth.nvfp4_tensor(64, 128, seed=2)
    p2 = str(tmp_path / "w.fp4c")
    makepad_b200.save_canonical(p2, _lib.FMT_NVFP4, b, sfb, 0.25)
    fmt, c3, s3, ts = makepad_b200.load_canonical(p2)
    assert fmt == _lib.FMT_NVFP4 and np.array_equal(c3, b) and np.array_equal(s3, sfb) and ts == 0.25
    info = _lib.FileInfo()
    assert _lib.load().mpq_file_info(p2.encode(), C.byref(info)) == _lib.OK
    assert (info.kind, info.N, info.K, info.bytes_a, info.bytes_b) == (_lib.FILE_CANONICAL, 64, 128, 64 * 64, 64 * 8)


def test_canonical_files_are_validated(tmp_path):
    import makepad_b200
    lib = _lib.load()
    codes, scales = synth.q4_weight(32, 64, seed=3)
    p = str(tmp_path / "w.q4c")
    makepad_b200.save_canonical(p, _lib.FMT_Q4, codes, scales)
    raw = bytearray(open(p, "rb").read())
    info = _lib.FileInfo()
    # a flipped payload byte: the checksum catches it
    bad = bytearray(raw); bad[200] ^= 0x40
    open(p, "wb").write(bad)
    with pytest.raises(makepad_b200.MpqError) as e:
        makepad_b200.load_canonical(p)
    assert e.value.status == _lib.ERR_FORMAT
    # truncated, wrong magic, future container version
    open(p, "wb").write(raw[:-1])
    assert lib.mpq_file_info(p.encode(), C.byref(info)) == _lib.ERR_FORMAT
    bad = bytearray(raw); bad[0] ^= 1
    open(p, "wb").write(bad)
    assert lib.mpq_file_info(p.encode(), C.byref(info)) == _lib.ERR_FORMAT
    bad = bytearray(raw); struct.pack_into("<I", bad, 4, 99)
    open(p, "wb").write(bad)
    assert lib.mpq_file_info(p.encode(), C.byref(info)) == _lib.ERR_FORMAT
    assert lib.mpq_file_info(str(tmp_path / "missing").encode(), C.byref(info)) == _lib.ERR_IO
    # capacity and shape checks
    open(p, "wb").write(raw)
    small = np.empty(8, dtype=np.uint8)
    assert lib.mpq_canonical_load(p.encode(), small.ctypes.data, small.nbytes, small.ctypes.data, small.nbytes, None) == _lib.ERR_SHAPE
    assert lib.mpq_canonical_save(p.encode(), _lib.FMT_Q4, 32, 48, codes.ctypes.data, scales.ctypes.data, C.c_float(1.0)) == _lib.ERR_SHAPE


@pytest.mark.gpu
def test_device_layout_roundtrip(ctx, orc, tmp_path):
    import torch
    import makepad_b200
    codes, scales = synth.q4_weight(1000, 2112, seed=4)
    w = makepad_b200.Q4Weight(ctx, codes, scales)
    p = str(tmp_path / "w.q4d")
    w.save(p)
    before = ctx.launches
    w2 = makepad_b200.load_weight(ctx, p)
    assert ctx.launches == before                                  # no repack kernel ran
    assert (w2.N, w2.K, w2.fmt) == (1000, 2112, _lib.FMT_Q4) and w2.device_bytes == w.device_bytes
    assert np.array_equal(w2.dequantize().cpu().numpy().view(np.uint32), orc.q4_dequantize(codes, scales).view(np.uint32))
    x = torch.from_numpy(synth.activations(3, 2112, seed=5)).cuda()
    assert torch.equal(makepad_b200.QuantLinear(w)(x), makepad_b200.QuantLinear(w2)(x))
    # NVFP4
    b, sfb = synth.nvfp4_tensor(448, 512, seed=6)
    w4 = makepad_b200.Nvfp4Weight(ctx, b, sfb, 0.5)
    p4 = str(tmp_path / "w.fp4d")
    w4.save(p4)
    w5 = makepad_b200.load_weight(ctx, p4)
    assert w5.tensor_scale == 0.5
    assert np.array_equal(w5.dequantize().cpu().numpy().view(np.uint32), orc.nvfp4_dequantize(b, sfb, 0.5).view(np.uint32))
    a, sfa = synth.nvfp4_tensor(200, 512, seed=7)
    ad, sd = torch.from_numpy(a).cuda(), torch.from_numpy(sfa).cuda()
    assert torch.equal(makepad_b200.QuantLinear(w4)((ad, sd, 1.0)).view(torch.int16), makepad_b200.QuantLinear(w5)((ad, sd, 1.0)).view(torch.int16))
    torch.cuda.synchronize()


@pytest.mark.gpu
def test_stale_or_damaged_cache_files_are_refused(ctx, tmp_path):
    import makepad_b200
    codes, scales = synth.q4_weight(64, 128, seed=8)
    w = makepad_b200.Q4Weight(ctx, codes, scales)
    p = str(tmp_path / "w.q4d")
    w.save(p)
    raw = bytearray(open(p, "rb").read())
    h = C.c_void_p()
    for mutate in ("layout", "payload", "truncate", "canonical"):
        bad = bytearray(raw)
        if mutate == "layout":
            struct.pack_into("<I", bad, 16, 1)                     # an older layout version
        elif mutate == "payload":
            bad[128 + 77] ^= 0x01
        elif mutate == "truncate":
            bad = bad[:-16]
        else:
            makepad_b200.save_canonical(p, _lib.FMT_Q4, codes, scales)
            bad = bytearray(open(p, "rb").read())
        open(p, "wb").write(bad)
        assert ctx.lib.mpq_weight_load(ctx.h, p.encode(), C.byref(h)) == _lib.ERR_FORMAT, mutate
        assert not h.value
    assert ctx.lib.mpq_weight_load(ctx.h, str(tmp_path / "nope").encode(), C.byref(h)) == _lib.ERR_IO


@pytest.mark.gpu
@pytest.mark.parametrize("N, K", [(1, 32), (33, 288), (96, 1216), (1000, 2112), (4097, 4096), (12320, 4096)])
def test_device_checksum_is_the_host_loop(ctx, tmp_path, N, K):
    """The checksum taken on the GPU against the host's byte loop over the same payload (just above one chunk of 4096 bytes, across
    chunks, across groups of 64 chunks, and across 64 groups), and a payload byte flipped anywhere is refused."""
    import makepad_b200
    w = makepad_b200.Q4Weight(ctx, *synth.q4_weight(N, K, seed=N))
    path, ref = str(tmp_path / "w.q4d"), str(tmp_path / "ref.q4c")
    w.save(path)
    raw = bytearray(open(path, "rb").read())
    payload = np.frombuffer(bytes(raw[128:]), dtype=np.uint8)
    # a tile stream of 1152-byte units is as long as the canonical arrays of the padded shape, whose file the host sums
    n, k = (N + 31) // 32 * 32, (K + 255) // 256 * 256
    cut = n * k // 2
    assert payload.size == n * k * 9 // 16
    makepad_b200.save_canonical(ref, _lib.FMT_Q4, payload[:cut].reshape(n, k // 2), payload[cut:].view(np.uint16).reshape(n, k // 32))
    assert raw[56:64] == open(ref, "rb").read()[56:64]
    want = w.dequantize()
    assert np.array_equal(makepad_b200.load_weight(ctx, path).dequantize().cpu().numpy(), want.cpu().numpy())
    for at in (128, len(raw) // 2, len(raw) - 1):
        bad = bytearray(raw)
        bad[at] ^= 0x80
        open(path, "wb").write(bad)
        with pytest.raises(makepad_b200.MpqError) as err:
            makepad_b200.load_weight(ctx, path)
        assert err.value.status == _lib.ERR_FORMAT


@pytest.mark.gpu
def test_a_weight_that_did_not_fit_does_not_fail_the_next_one(ctx, tmp_path):
    """A creation that finds no device memory reports it once: the error is not left behind for the next creation, load or export."""
    import makepad_b200
    codes, scales = synth.q4_weight(96, 1216, seed=5)
    path = str(tmp_path / "w.q4d")
    makepad_b200.Q4Weight(ctx, codes, scales).save(path)
    h = C.c_void_p()

    def too_large():                                                   # 2^40 weights: 618 GB, refused before an array is read
        assert ctx.lib.mpq_q4_weight_create(ctx.h, 1 << 20, 1 << 20, codes.ctypes.data, scales.ctypes.data, _lib.TP_NONE, 0, 1, C.byref(h)) == _lib.ERR_CUDA
        assert not h.value

    too_large()
    w = makepad_b200.Q4Weight(ctx, codes, scales)
    want = w.dequantize().cpu().numpy()
    too_large()
    assert np.array_equal(makepad_b200.load_weight(ctx, path).dequantize().cpu().numpy(), want)
    too_large()
    assert np.array_equal(w.dequantize().cpu().numpy(), want)
    too_large()
    w.save(path)


@pytest.mark.gpu
def test_save_and_load_need_no_device_memory_beside_the_weight(ctx, tmp_path):
    """The checksum wants 1/32 of the weight's bytes on the device; without them it is taken on the host."""
    import torch
    import makepad_b200
    N, K = 32768, 16384                                                # 302 MB, 9.4 MB for the checksum
    codes = np.random.default_rng(7).integers(0, 256, (N, K // 2), dtype=np.uint8)
    scales = np.full((N, K // 32), 0x2C00, dtype=np.uint16)
    path, full = str(tmp_path / "w.q4d"), str(tmp_path / "full.q4d")
    c2 = makepad_b200.Context(0)                                       # (its upload has kept no memory that would do)
    w = makepad_b200.Q4Weight(ctx, codes, scales)
    w.save(path)

    def hold(left):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")

    held = hold(4 << 20)
    assert c2.lib.mpq_weight_save(c2.h, w.h, full.encode()) == _lib.OK
    assert open(full, "rb").read() == open(path, "rb").read()
    w.destroy()
    del held
    held = hold((N * K * 9 // 16) + (6 << 20))
    back = makepad_b200.load_weight(c2, full)
    h = C.c_void_p()
    back.destroy()
    with open(full, "r+b") as f:                                       # and a damaged file is still found out
        f.seek(128 + 12345678)
        byte = f.read(1)[0]
        f.seek(128 + 12345678)
        f.write(bytes([byte ^ 1]))
    assert c2.lib.mpq_weight_load(c2.h, full.encode(), C.byref(h)) == _lib.ERR_FORMAT and not h.value
    del held
    torch.cuda.empty_cache()
    back = makepad_b200.load_weight(c2, path)
    back.save(full)
    assert open(full, "rb").read() == open(path, "rb").read()
    back.destroy()
    c2.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["page-locked", "half page-locked", "pageable", "device"])
def test_weights_from_every_kind_of_memory(ctx, kind):
    """Arrays that the driver reads by itself and arrays that go through the pinned slots give the same weight."""
    import torch
    import makepad_b200
    N, K = 3000, 2112                                                  # 3.2 MB of codes: several slots
    codes, scales = synth.q4_weight(N, K, seed=91)
    want = makepad_b200.Q4Weight(ctx, codes, scales).dequantize()
    c, s = torch.from_numpy(codes), torch.from_numpy(scales.view(np.int16))
    registered = 0
    if kind == "page-locked":
        c, s = c.pin_memory(), s.pin_memory()
    elif kind == "half page-locked":                                   # the first of the array's pages
        c = c.clone()
        registered = (c.data_ptr() + 4095) // 4096 * 4096
        assert int(torch.cuda.cudart().cudaHostRegister(registered, 1 << 20, 0)) == 0
    elif kind == "device":
        c, s = c.cuda(), s.cuda()
    h = C.c_void_p()
    ctx.check(ctx.lib.mpq_q4_weight_create(ctx.h, N, K, c.data_ptr(), s.data_ptr(), _lib.TP_NONE, 0, 1, C.byref(h)))
    if registered:
        assert int(torch.cuda.cudart().cudaHostUnregister(registered)) == 0
    out = torch.empty_like(want)
    ctx.check(ctx.lib.mpq_weight_dequantize(ctx.h, h, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int32), want.view(torch.int32))
    ctx.lib.mpq_weight_destroy(h)


def _fnv1a64(data):
    h = 0xCBF29CE484222325
    for b in data:
        h = (h ^ b) * 0x100000001B3 & 0xFFFFFFFFFFFFFFFF
    return h


@pytest.mark.gpu
@pytest.mark.parametrize("N, K", [(8, 32), (8, 96), (24, 4096), (232, 544), (248, 4128)])
def test_device_checksum_continues_from_the_codes_to_the_scale_factors(ctx, tmp_path, N, K):
    """NVFP4 files have two parts: the stored checksum is that of a plain loop over both.  The codes are less than one chunk of 4096
    bytes, whole chunks, and more than a group of 64 chunks with a ragged end; a flipped byte in either part is refused."""
    import makepad_b200
    w = makepad_b200.Nvfp4Weight(ctx, *synth.nvfp4_tensor(N, K, seed=N + K), 0.5)
    path = str(tmp_path / "w.fp4d")
    w.save(path)
    raw = bytearray(open(path, "rb").read())
    assert len(raw) > 128 + N * K // 2
    assert int.from_bytes(raw[56:64], "little") == _fnv1a64(raw[128:])
    want = w.dequantize()
    assert np.array_equal(makepad_b200.load_weight(ctx, path).dequantize().cpu().numpy(), want.cpu().numpy())
    for at in (128, 128 + N * K // 2 - 1, 128 + N * K // 2, len(raw) - 1):
        bad = bytearray(raw)
        bad[at] ^= 1
        open(path, "wb").write(bad)
        with pytest.raises(makepad_b200.MpqError) as err:
            makepad_b200.load_weight(ctx, path)
        assert err.value.status == _lib.ERR_FORMAT


@pytest.mark.gpu
def test_page_locked_arrays_that_are_still_being_written(ctx):
    """Arrays that an asynchronous copy on the default stream fills: the upload follows that copy, as cudaMemcpy does."""
    import torch
    import makepad_b200
    N, K = 1000, 2112
    codes, scales = synth.q4_weight(N, K, seed=92)
    want = makepad_b200.Q4Weight(ctx, codes, scales).dequantize()
    cd, sd = torch.from_numpy(codes).cuda(), torch.from_numpy(scales.view(np.int16)).cuda()
    c, s = torch.zeros_like(cd, device="cpu").pin_memory(), torch.zeros_like(sd, device="cpu").pin_memory()
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)                                     # a tenth of a second
    c.copy_(cd, non_blocking=True)
    s.copy_(sd, non_blocking=True)
    w = makepad_b200.Q4Weight(ctx, c.numpy(), s.numpy().view(np.uint16))
    assert torch.equal(w.dequantize().view(torch.int32), want.view(torch.int32))


@pytest.mark.gpu
def test_first_call_on_a_side_stream_finds_its_slots_empty(orc):
    """The streaming kernel's slots are cleared when they are made; the first launch, on a stream that does not wait for the default
    one, must find them cleared although their memory held something else before."""
    import torch
    import makepad_b200
    N, K = 1000, 11008                                                 # row tiles that several CTAs share
    codes, scales = synth.q4_weight(N, K, seed=93)
    x = synth.activations(1, K, seed=94)
    ref = orc.q4_matmul_f64(codes, scales, x)
    side = torch.cuda.Stream()
    xd = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    for _ in range(8):
        dirt = [torch.full((1 << 18,), 1.0, device="cuda") for _ in range(16)]
        torch.cuda.synchronize()
        del dirt
        torch.cuda.empty_cache()                                       # back to the driver: the next slots may lie there
        c2 = makepad_b200.Context(0)
        lin = makepad_b200.QuantLinear(makepad_b200.Q4Weight(c2, codes, scales))
        with torch.cuda.stream(side):
            y = lin(xd)
        side.synchronize()
        assert orc.err_report(y.cpu().numpy(), ref)["max_abs_over_rms"] < 2e-5
        assert c2.lib.mpq_context_poll_status(c2.h) == _lib.OK
        del lin
        c2.close()
