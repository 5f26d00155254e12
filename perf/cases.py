"""The work that is timed on this package: what a serving process and a checkpoint loader have it do.

`listed()` names the cases, `draw(rng)` makes one more of the same ranges, `prepare` builds what a program holds before
the call (weights in the kernels' format, inputs, a captured CUDA graph where such a program replays one), `run` is one
pass through the package's public functions, `work` the bytes and operations such a pass cannot do without, `tolerance`
how far another correct implementation of the same precision may be from it.

Activations are N(0, 1) in bf16, weights N(0, 0.02) in fp32 quantized to E4M3 with 128x128 block scales (the value
distributions of the package's benchmark); everything is made on the GPU from the seed.
"""

import math

import torch

import gaudi_kernels_b200 as gk
from gaudi_kernels_b200.block_fp8_gemm import new_status

DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
BLOCK = 128

# A drawn case costs no more than the largest listed one: the prefill FFN below, 3 * 2 * 8192 * 4096 * 14336 operations
MAX_FLOPS = 3 * 2 * 8192 * 4096 * 14336
MAX_CODEC_ELEMS = 8192 * 8192
MAX_WEIGHT_ELEMS = 28672 * 4096


def listed():
    return [
        # one token through one projection, called eagerly: 59 MB of weight, so launches and host time count
        {"name": "linear_decode_m1", "kind": "linear", "m": 1, "k": 4096, "n": 14336, "half": True, "out": "bf16", "bias": False},
        # a decode step's whole FFN as a server replays it: a CUDA graph of quantize, gate/up + SwiGLU, quantize, down
        {"name": "ffn_decode_m8", "kind": "ffn", "m": 8, "k": 4096, "inter": 14336, "graph": True},
        {"name": "ffn_decode_m64", "kind": "ffn", "m": 64, "k": 4096, "inter": 14336, "graph": True},
        # a chunk of a prompt (or a large decode batch) through a square projection; the row count is what arrived
        {"name": "linear_chunk_m300", "kind": "linear", "m": 300, "k": 4096, "n": 4096, "half": True, "out": "bf16", "bias": True},
        # the long-K projection (FFN down) for a chunk of 512 rows
        {"name": "linear_down_m512", "kind": "linear", "m": 512, "k": 14336, "n": 4096, "half": True, "out": "bf16", "bias": False},
        # odd sizes in every dimension, fp32 result, OCP codes as the checkpoint stores them
        {"name": "linear_ragged", "kind": "linear", "m": 777, "k": 1000, "n": 1003, "half": False, "out": "f32", "bias": True},
        # a whole prompt batch through the FFN: the largest case
        {"name": "ffn_prefill_m8192", "kind": "ffn", "m": 8192, "k": 4096, "inter": 14336, "graph": False},
        # the per-token / per-channel variant, decode batch and prefill
        {"name": "token_decode_m16", "kind": "token", "m": 16, "k": 4096, "n": 14336, "out": "bf16", "bias": False},
        {"name": "token_prefill_m4096", "kind": "token", "m": 4096, "k": 4096, "n": 14336, "out": "bf16", "bias": True},
        # weights to codes and back: the 128x128 quantizer and the decoder on the codec configuration
        {"name": "codec_8192", "kind": "codec", "rows": 8192, "cols": 8192, "half": True, "out": "bf16"},
        # loading a fused gate/up weight: half-range re-encode with its checks, then the layout of the fused GEMM
        {"name": "load_gate_up", "kind": "load", "rows": 28672, "k": 4096, "swiglu": True},
        # the reference's own call on host tensors: upload, re-encode, quantize, multiply, copy back
        {"name": "reference_host_m1024", "kind": "host", "m": 1024, "k": 4096, "n": 14336, "half": True},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _size(rng, lo, hi):
    """A projection's width: mostly a multiple of the scale block, sometimes of 16, sometimes any number."""
    v = _log_int(rng, lo, hi)
    step = rng.choice((BLOCK, BLOCK, BLOCK, 16, 1))
    return max(step, v // step * step)


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear", "ffn", "ffn", "token", "codec", "load", "host"))
    while True:
        if kind == "linear":
            c = {"kind": kind, "m": _log_int(rng, 1, 8192), "k": _size(rng, 512, 14336), "n": _size(rng, 512, 28672),
                 "half": rng.random() < 0.7, "out": rng.choice(("bf16", "bf16", "bf16", "f32")), "bias": rng.random() < 0.4}
        elif kind == "ffn":
            m = _log_int(rng, 1, 8192)
            c = {"kind": kind, "m": m, "k": _size(rng, 512, 8192), "inter": _log_int(rng, 1024, 14336) // BLOCK * BLOCK,
                 "graph": m <= 128}
        elif kind == "token":
            c = {"kind": kind, "m": _log_int(rng, 1, 8192), "k": _size(rng, 512, 14336), "n": _size(rng, 512, 14336),
                 "out": "bf16", "bias": rng.random() < 0.4}
        elif kind == "codec":
            c = {"kind": kind, "rows": _size(rng, 128, 16384), "cols": _size(rng, 128, 16384),
                 "half": rng.random() < 0.5, "out": rng.choice(("bf16", "f32"))}
        elif kind == "load":
            swiglu = rng.random() < 0.5
            rows = _log_int(rng, 1024, 28672) // 256 * 256 if swiglu else _size(rng, 1024, 28672)
            c = {"kind": kind, "rows": rows, "k": _size(rng, 512, 8192), "swiglu": swiglu}
        else:
            c = {"kind": kind, "m": _log_int(rng, 1, 2048), "k": _size(rng, 512, 4096), "n": _size(rng, 512, 14336),
                 "half": rng.random() < 0.7}
        if kind == "codec" and c["rows"] * c["cols"] > MAX_CODEC_ELEMS:
            continue
        if kind == "load" and c["rows"] * c["k"] > MAX_WEIGHT_ELEMS:
            continue
        if kind in ("linear", "ffn", "token", "host") and work(c)["flops"] > MAX_FLOPS:
            continue
        return c


def _activations(gen, m, k):
    return torch.randn((m, k), generator=gen, device="cuda").to(torch.bfloat16)


def _checkpoint_weight(gen, n, k):
    """OCP E4M3 codes and 128x128 scales of an N(0, 0.02) weight, as a checkpoint holds them."""
    return gk.quantize_block128(torch.randn((n, k), generator=gen, device="cuda") * 0.02)


def _bias(gen, n):
    return torch.randn((n,), generator=gen, device="cuda") * 0.1


_graph_stream = []


def _capture(fn):
    """fn's CUDA graph and its static outputs, warmed up and captured on one stream of this module."""
    if not _graph_stream:
        _graph_stream.append(torch.cuda.Stream())
    stream = _graph_stream[0]
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        fn()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = fn()
    return graph, out


def _ffn(s):
    codes, scales = gk.quantize_act_1x128(s["x"], native_half=True)
    h = gk.gemm_block_fp8_swiglu(codes, scales, s["gu"], s["gu_scales"], check=False)
    codes, scales = gk.quantize_act_1x128(h, native_half=True)
    return gk.gemm_block_fp8(codes, scales, s["down"], s["down_scales"], check=False, status=s["status"])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = dict(case)
    s["case"] = case
    if kind in ("linear", "ffn"):
        s["status"] = new_status(torch.device("cuda", torch.cuda.current_device()))
    if kind == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        s["x"] = _activations(gen, m, k)
        s["w"], s["w_scales"] = gk.prepare_weight(*_checkpoint_weight(gen, n, k), native_half=case["half"])
        s["bias"] = _bias(gen, n) if case["bias"] else None
    elif kind == "ffn":
        m, k, inter = case["m"], case["k"], case["inter"]
        s["x"] = _activations(gen, m, k)
        s["gu"], s["gu_scales"] = gk.prepare_weight_swiglu(*_checkpoint_weight(gen, 2 * inter, k))
        s["down"], s["down_scales"] = gk.prepare_weight(*_checkpoint_weight(gen, k, inter))
        if case["graph"]:
            # a server declares its weights at rest once the checkpoint is loaded; the captured launches keep that
            torch.cuda.synchronize()
            before = gk.set_weights_at_rest(True)
            try:
                s["graph"], s["y"] = _capture(lambda: _ffn(s))
            finally:
                gk.set_weights_at_rest(before)
        else:
            s["graph"] = None
    elif kind == "token":
        m, k, n = case["m"], case["k"], case["n"]
        s["x"] = _activations(gen, m, k)
        w = torch.randn((n, k), generator=gen, device="cuda") * 0.02
        s["w_scales"] = w.abs().amax(1) / 448.0                       # one scale per output channel
        s["w"] = (w / s["w_scales"][:, None]).to(torch.float8_e4m3fn)
        s["bias"] = _bias(gen, n) if case["bias"] else None
    elif kind == "codec":
        w = torch.randn((case["rows"], case["cols"]), generator=gen, device="cuda") * 0.02
        spikes = torch.rand(w.shape, generator=gen, device="cuda") < 0.001
        s["w"] = torch.where(spikes, w * 50.0, w)
    elif kind == "load":
        s["w"], s["w_scales"] = _checkpoint_weight(gen, case["rows"], case["k"])
    else:
        s["x"] = _activations(gen, case["m"], case["k"]).cpu().pin_memory()
        w, ws = _checkpoint_weight(gen, case["n"], case["k"])
        s["w"], s["w_scales"] = w.cpu().pin_memory(), ws.cpu().pin_memory()
        s["y"] = torch.empty((case["m"], case["n"]), dtype=torch.bfloat16).pin_memory()
    return s


def run(s):
    kind = s["kind"]
    if kind == "linear":
        codes, scales = gk.quantize_act_1x128(s["x"], native_half=s["half"])
        return gk.gemm_block_fp8(codes, scales, s["w"], s["w_scales"], bias=s["bias"], out_dtype=DTYPES[s["out"]],
                                 check=False, status=s["status"])
    if kind == "ffn":
        if s["graph"] is None:
            return _ffn(s)
        s["graph"].replay()
        return s["y"]
    if kind == "token":
        codes, scales = gk.quantize_act_token(s["x"], native_half=True)
        return gk.gemm_token_channel_fp8(codes, scales, s["w"], s["w_scales"], bias=s["bias"],
                                         out_dtype=DTYPES[s["out"]], check=False)
    if kind == "codec":
        codes, scales = gk.quantize_block128(s["w"], native_half=s["half"])
        return codes, scales, gk.decode_e4m3(codes, scales, out_dtype=DTYPES[s["out"]])
    if kind == "load":
        if s["swiglu"]:
            return gk.prepare_weight_swiglu(s["w"], s["w_scales"])
        return gk.reencode_e4m3fn_half(s["w"], s["w_scales"])
    return gk.reference(s["x"], s["w"], s["w_scales"], native_half=s["half"], out=s["y"])


def _blocks(n):
    return (n + BLOCK - 1) // BLOCK


def work(case):
    """Inputs read once, outputs written once, and 2 operations per multiply-add of the products."""
    kind = case["kind"]
    if kind in ("linear", "host"):
        m, k, n = case["m"], case["k"], case["n"]
        out = 4 if case.get("out") == "f32" else 2
        return {"bytes": 2 * m * k + n * k + 4 * _blocks(n) * _blocks(k) + (4 * n if case.get("bias") else 0) + out * m * n,
                "flops": 2 * m * n * k}
    if kind == "ffn":
        m, k, inter = case["m"], case["k"], case["inter"]
        return {"bytes": 2 * m * k + 3 * inter * k + 4 * 3 * _blocks(inter) * _blocks(k) + 2 * m * k,
                "flops": 3 * 2 * m * k * inter}
    if kind == "token":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 2 * m * k + n * k + 4 * n + (4 * n if case["bias"] else 0) + 2 * m * n, "flops": 2 * m * n * k}
    if kind == "codec":
        elems, grid = case["rows"] * case["cols"], _blocks(case["rows"]) * _blocks(case["cols"])
        return {"bytes": (4 + 1 + (4 if case["out"] == "f32" else 2)) * elems + 4 * grid, "flops": 2 * elems}
    elems, grid = case["rows"] * case["k"], _blocks(case["rows"]) * _blocks(case["k"])
    return {"bytes": 2 * elems + 8 * grid, "flops": elems}


def tolerance(case):
    """Relative 2-norm error of another correct implementation, measured against sums in 64 bits.

    fp32 results differed by 0.7e-7 to 1.4e-7 (K from 1000 to 7296; longer sums have more roundings).  bf16 results are
    the same sums rounded once: a few in a thousand fall to the other neighbour, 1e-5 to 4e-5 over a large result, up to
    4e-4 where one of only 512 values does.  In the FFN such a value can also change an E4M3 code of the intermediate:
    0.3e-5 to 2.3e-4 measured, more for the narrowest ones.
    """
    kind = case["kind"]
    if kind in ("codec", "load"):
        return "exact"
    if kind == "ffn":
        return {"rel": 3e-3}
    return {"rel": 1e-3 if case.get("out", "bf16") == "bf16" else 1e-6}
