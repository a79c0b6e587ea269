"""The work that programs built on this library have it do, as timed cases.

A case is a dict of plain values with a "kind":

  q4         y = x . W^T through QuantLinear on a Q4 weight, M fp32 activation rows on the GPU
  q4_host    the same call on host arrays (numpy in, numpy out: the library copies)
  q4_ffn     gate+up projection, then the down projection with SwiGLU fused in front (a feed-forward block)
  q4_stack   one decode / tree-verify step of the 7B-shape projection stack, replayed as a CUDA graph
  nvfp4      quantise M activation rows to NVFP4, then the block-scaled GEMM (bf16 out)
  nvfp4_ffn  a feed-forward block in NVFP4: quantise, gate+up GEMM, SwiGLU + quantise, down GEMM
  pack       Q4 weight from host arrays in the interchange format, and its exact fp32 export
  load       a weight file in the device layout, read back into device memory, and its export

Sizes are the 7B / 70B projection shapes of the benchmark and the ragged ones of the tests; distributions are the
benchmark's: codes uniform, Q4 scales fp16(|N(0,1)| * 0.02), NVFP4 scales e4m3(|N(0,1)| * 0.1), activations N(0,1).
"""
import math
import os
import tempfile

import torch

import makepad_b200 as mpq
from makepad_b200.decode_stack import SHAPES_7B, DecodeStack

_context = []


def context():
    """One library context per process, as a program keeps it."""
    if not _context:
        _context.append(mpq.Context(0))
    return _context[0]


def listed():
    return [
        # one projection of one token: the smallest call, where latency counts
        {"name": "q4 matvec 4096x4096", "kind": "q4", "M": 1, "N": 4096, "K": 4096},
        # one token through all 32 layers' projections: the decode step
        {"name": "q4 decode step 7B", "kind": "q4_stack", "M": 1, "layers": 32},
        # eight drafted tokens verified at once (the middle of the verify widths 2, 4, 8, 16)
        {"name": "q4 verify 8 rows 7B", "kind": "q4_stack", "M": 8, "layers": 4},
        # a few sequences decoded together through a small matrix of no round size
        {"name": "q4 ragged 13 rows", "kind": "q4", "M": 13, "N": 1000, "K": 2112},
        # 64 sequences decoded together: the feed-forward block of the 70B shape
        {"name": "q4 ffn 70B 64 rows", "kind": "q4_ffn", "M": 64, "H": 8192, "F": 28672},
        # a prompt through a model whose weights are Q4: the feed-forward block of the 7B shape
        {"name": "q4 ffn 7B prompt 512", "kind": "q4_ffn", "M": 512, "H": 4096, "F": 11008},
        # a caller with host buffers: the QKV projection of one token
        {"name": "q4 host qkv 1 row", "kind": "q4_host", "M": 1, "N": 12288, "K": 4096},
        # NVFP4 weights at decode time: 16 sequences, bf16 activations
        {"name": "nvfp4 16 rows", "kind": "nvfp4", "M": 16, "N": 14336, "K": 4096, "dtype": "bf16"},
        # NVFP4 prefill: the GEMM configuration of the benchmark, from bf16 activations
        {"name": "nvfp4 prefill 2048", "kind": "nvfp4", "M": 2048, "N": 14336, "K": 4096, "dtype": "bf16"},
        # a prompt of no round length through a whole NVFP4 feed-forward block, from fp32 activations
        {"name": "nvfp4 ffn prompt 1000", "kind": "nvfp4_ffn", "M": 1000, "H": 4096, "F": 14336, "dtype": "fp32"},
        # start-up from interchange arrays: one layer's QKV weight packed on the GPU
        {"name": "q4 pack qkv", "kind": "pack", "N": 12288, "K": 4096},
        # start-up from the cache file of the same weight
        {"name": "q4 load qkv", "kind": "load", "N": 12288, "K": 4096},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step`, its logarithm uniform over lo..hi."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["q4", "q4", "q4_host", "q4_ffn", "q4_ffn", "q4_stack", "nvfp4", "nvfp4", "nvfp4_ffn", "pack", "load"])
    if kind in ("q4", "q4_host"):
        # any N, any K that is a multiple of 32; decode batches mostly, prompts too
        n, k = _log(rng, 500, 30000), _log(rng, 512, 12288, 32)
        most = min(512, 6 * 10 ** 10 // (n * k)) if kind == "q4" else 32
        c = {"kind": kind, "M": _log(rng, 1, most), "N": n, "K": k}
    elif kind == "q4_ffn":
        h = _log(rng, 1024, 8192, 64)
        c = {"kind": kind, "M": _log(rng, 1, 512 if h <= 4096 else 64), "H": h, "F": int(h * rng.uniform(2.5, 3.5)) // 32 * 32}
    elif kind == "q4_stack":
        c = {"kind": kind, "M": _log(rng, 1, 64), "layers": rng.randint(1, 8)}
    elif kind == "nvfp4":
        n, k = _log(rng, 1024, 16384, 8), _log(rng, 1024, 8192, 32)
        c = {"kind": kind, "M": _log(rng, 1, min(4096, 12 * 10 ** 10 // (n * k))), "N": n, "K": k, "dtype": rng.choice(["bf16", "fp32"])}
    elif kind == "nvfp4_ffn":
        h = _log(rng, 1024, 4096, 64)
        c = {"kind": kind, "M": _log(rng, 1, 1000), "H": h, "F": int(h * rng.uniform(2.5, 3.5)) // 32 * 32, "dtype": rng.choice(["bf16", "fp32"])}
    else:
        c = {"kind": kind, "N": _log(rng, 500, 16384), "K": _log(rng, 512, 8192, 32)}
    return c


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _q4_arrays(g, n, k):
    codes = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    scales = (torch.randn((n, k // 32), device="cuda", generator=g).abs() * 0.02).to(torch.float16).view(torch.int16)
    return codes.cpu().numpy(), scales.cpu().numpy().view("uint16")


def _q4_linear(g, n, k):
    return mpq.QuantLinear(mpq.Q4Weight(context(), *_q4_arrays(g, n, k)))


def _nvfp4_linear(g, n, k):
    codes = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    sf = (torch.randn((n, k // 16), device="cuda", generator=g).abs() * 0.1).to(torch.float8_e4m3fn).view(torch.uint8)
    # the tensor scale brings the outputs back to the size of the inputs (the codes' rms is about 3, the scales' 0.1)
    return mpq.QuantLinear(mpq.Nvfp4Weight(context(), codes.cpu().numpy(), sf.cpu().numpy(), 3.2 / math.sqrt(k)))


def _rows(g, m, k, dtype="fp32"):
    return torch.randn((m, k), device="cuda", generator=g).to(torch.bfloat16 if dtype == "bf16" else torch.float32)


class _File:
    """A weight file of this process, gone with the object."""

    def __init__(self):
        fd, self.path = tempfile.mkstemp(suffix=".mpq")
        os.close(fd)

    def __del__(self):
        try:
            os.unlink(self.path)
        except OSError:
            pass


def prepare(case, seed):
    g, kind, s = _gen(seed), case["kind"], dict(case)
    if kind == "q4_stack":
        s["stack"] = DecodeStack(context(), layers=case["layers"], M=case["M"], shapes=SHAPES_7B, seed=seed * 1009 % (1 << 40)).capture()
    elif kind in ("q4", "q4_host"):
        s["linear"] = _q4_linear(g, case["N"], case["K"])
        s["x"] = _rows(g, case["M"], case["K"])
        if kind == "q4_host":
            s["x"] = s["x"].cpu().numpy()
    elif kind == "q4_ffn":
        s["gate_up"], s["down"] = _q4_linear(g, 2 * case["F"], case["H"]), _q4_linear(g, case["H"], case["F"])
        s["x"] = _rows(g, case["M"], case["H"])
    elif kind == "nvfp4":
        s["linear"] = _nvfp4_linear(g, case["N"], case["K"])
        s["x"] = _rows(g, case["M"], case["K"], case["dtype"])
    elif kind == "nvfp4_ffn":
        s["gate_up"], s["down"] = _nvfp4_linear(g, 2 * case["F"], case["H"]), _nvfp4_linear(g, case["H"], case["F"])
        s["x"] = _rows(g, case["M"], case["H"], case["dtype"])
    elif kind == "pack":
        s["codes"], s["scales"] = _q4_arrays(g, case["N"], case["K"])
    elif kind == "load":
        s["file"] = _File()
        w = mpq.Q4Weight(context(), *_q4_arrays(g, case["N"], case["K"]))
        w.save(s["file"].path)
        w.destroy()
    return s


def run(s):
    kind = s["kind"]
    if kind == "q4_stack":
        s["stack"].step()
        return s["stack"].y
    if kind in ("q4", "q4_host"):
        return s["linear"](s["x"])
    if kind == "q4_ffn":
        return s["down"].forward_swiglu(s["gate_up"](s["x"]))
    if kind == "nvfp4":
        codes, sf = mpq.nvfp4_quantize(context(), s["x"])
        return s["linear"]((codes, sf, 1.0))
    if kind == "nvfp4_ffn":
        codes, sf = mpq.nvfp4_quantize(context(), s["x"])
        hidden = s["gate_up"]((codes, sf, 1.0))
        codes, sf = mpq.nvfp4_quantize(context(), hidden, swiglu_fused=True)
        return s["down"]((codes, sf, 1.0))
    # the weight of the pass before is given up when the new one is there, as on a reload
    if kind == "pack":
        s["weight"] = mpq.Q4Weight(context(), s["codes"], s["scales"])
    else:
        s["weight"] = mpq.load_weight(context(), s["file"].path)
    return s["weight"].dequantize()


def _q4_work(m, n, k):
    return n * k * 9 // 16 + 4 * m * (n + k), 2 * m * n * k


def work(case):
    kind, m = case["kind"], case.get("M")
    size = 2 if case.get("dtype") == "bf16" else 4
    if kind == "q4_stack":
        parts = [_q4_work(m, n, k) for _, n, k in SHAPES_7B] * case["layers"]
    elif kind in ("q4", "q4_host"):
        parts = [_q4_work(m, case["N"], case["K"])]
    elif kind == "q4_ffn":
        h, f = case["H"], case["F"]
        parts = [_q4_work(m, 2 * f, h), _q4_work(m, h, f), (4 * m * f, 0)]     # the down projection reads gate and up
    elif kind == "nvfp4":
        n, k = case["N"], case["K"]
        parts = [(n * k * 9 // 16 + size * m * k + 2 * m * n, 2 * m * n * k)]
    elif kind == "nvfp4_ffn":
        h, f = case["H"], case["F"]
        parts = [(size * m * h + 2 * m * h + 3 * f * h * 9 // 16, 6 * m * h * f)]
    else:                                            # interchange arrays or file in, device layout, fp32 export out
        n, k = case["N"], case["K"]
        parts = [(2 * (n * k * 9 // 16) + 4 * n * k, n * k)]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("pack", "load"):
        return "exact"
    if kind.startswith("q4"):
        return {"rel": 1e-5, "max": 1e-4}            # fp32 sums of products that are exact to 22 bits
    if kind == "nvfp4":
        return {"rel": 5e-3, "max": 2e-2}            # bf16 results of fp32 sums
    return {"rel": 1e-2, "max": 0.3}                 # a bf16 ulp of the hidden layer can move a 4-bit code of the next GEMM's input
