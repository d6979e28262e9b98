"""The work whose speed this framework is judged by: Matmul nodes as the models behind it run them.

Each case is one pass through the public entry points (Linear, MLP, Executable, Tensor.gemm / resolve / to) at the sizes
of the repository's configurations, tests and benchmark:

    lazy       Linears scheduled one after the other, resolved, and the last output read back to the host
    decode     one token through the MLPs of all layers, bound once as one Executable
    mlp        MLP blocks (fc1, activation, fc2), each with an input of its own, one MLP.schedule each
    linear     one dense f32 Linear as an Executable
    attention  the two products of an attention layer, q.kT and softmax.v, as one Executable

Weights are N(0, 1/K) so that activations keep the scale they have behind a normalisation; they are quantised on the GPU
with the formats' own rules.  Everything is made from the seed.
"""
import math
import types

import numpy as np
import torch

import ratchet_b200 as rb
from ratchet_b200 import Device, DeviceRequest, DType, Executable, GpuBuffer, Linear, MLP, Tensor

BYTES = {"F32": 4.0, "F16": 2.0, "BF16": 2.0, "Q8_0H": 34 / 32, "Q8_0F": 36 / 32, "Q4_K": 144 / 256}
TORCH = {"F32": torch.float32, "F16": torch.float16, "BF16": torch.bfloat16}


def listed():
    return [
        # one attention projection of Phi-2 called by itself on one token: the smallest call a program makes
        {"name": "linear_1row", "kind": "lazy", "weights": "Q8_0H", "layers": 0, "d": 2560, "ff": 0, "vocab": 2560, "rows": 1},
        # one token of Whisper-tiny's decoder (projection, fc1 + GELU, fc2 per layer, then the logits), as a lazy graph
        {"name": "whisper_token_lazy", "kind": "lazy", "weights": "Q8_0H", "layers": 4, "d": 384, "ff": 1536, "vocab": 51865, "rows": 1},
        # one token through Phi-2's 32 MLPs: the headline decode step
        {"name": "phi2_decode_q8", "kind": "decode", "weights": "Q8_0H", "layers": 32, "d": 2560, "ff": 10240},
        # the same on the default quantisation pair (f32 scales, f32 activations)
        {"name": "phi2_decode_q8f_f32", "kind": "decode", "weights": "Q8_0F", "layers": 8, "d": 2560, "ff": 10240},
        # one token through Phi-3-mini's gated MLPs with 4-bit weights
        {"name": "phi3_decode_q4k", "kind": "mlp", "weights": "Q4_K", "act": "silu_gate", "dtype": "F16", "blocks": 8, "d": 3072, "ff": 8192,
         "batch": 1, "rows": 1, "bias": False},
        # sixteen streams decoded together
        {"name": "phi3_batch16_q8", "kind": "mlp", "weights": "Q8_0H", "act": "silu_gate", "dtype": "F16", "blocks": 4, "d": 3072, "ff": 8192,
         "batch": 1, "rows": 16, "bias": False},
        # a short prompt of ragged length
        {"name": "phi2_prompt77_q8", "kind": "mlp", "weights": "Q8_0H", "act": "gelu", "dtype": "F16", "blocks": 4, "d": 2560, "ff": 10240,
         "batch": 1, "rows": 77, "bias": True},
        # the four encoder MLPs of Whisper-tiny over 30 s of audio
        {"name": "whisper_encoder_mlp", "kind": "mlp", "weights": "Q8_0H", "act": "gelu", "dtype": "F16", "blocks": 4, "d": 384, "ff": 1536,
         "batch": 1, "rows": 1500, "bias": True},
        # an ordinary prompt with 4-bit weights
        {"name": "phi3_prompt512_q4k", "kind": "mlp", "weights": "Q4_K", "act": "silu_gate", "dtype": "F16", "blocks": 4, "d": 3072, "ff": 8192,
         "batch": 1, "rows": 512, "bias": False},
        # a batch of long prompts in bf16: the largest
        {"name": "phi2_prefill_bf16", "kind": "mlp", "weights": "Q8_0H", "act": "gelu", "dtype": "BF16", "blocks": 1, "d": 2560, "ff": 10240,
         "batch": 4, "rows": 2048, "bias": True},
        # unquantised f32 weights
        {"name": "dense_f32_128", "kind": "linear", "d": 2560, "out": 10240, "rows": 128},
        # the attention products of Phi-2 over a 512-token prompt: scores in f32, values in f16
        {"name": "phi2_attention_512", "kind": "attention", "heads": 32, "dim": 80, "rows": 512, "context": 512, "scores": "F32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(v, m):
    return max(m, int(round(v / m)) * m)


def draw(rng):
    kind = rng.choice(["lazy", "decode", "decode", "mlp", "mlp", "mlp", "mlp", "mlp", "linear", "attention"])
    if kind == "lazy":
        w = rng.choice(["Q8_0H", "Q8_0H", "Q4_K", "F16"])
        step = 256 if w == "Q4_K" else 32
        d = _multiple(_log(rng, 384, 3072), step)
        layers = rng.randint(0, 6)
        return {"kind": "lazy", "weights": w, "layers": layers, "d": d, "ff": _multiple(d * rng.uniform(2.5, 4), step) if layers else 0,
                "vocab": _log(rng, 1001, 51865), "rows": rng.choice([1, 1, 1, 2, 5])}
    if kind == "decode":
        w = rng.choice(["Q8_0H", "Q8_0H", "Q8_0F"])
        d = _multiple(_log(rng, 1024, 3072), 32)
        return {"kind": "decode", "weights": w, "layers": _log(rng, 2, 24), "d": d, "ff": _multiple(d * rng.uniform(2.5, 4), 32)}
    if kind == "mlp":
        w = rng.choice(["Q8_0H", "Q8_0H", "Q4_K", "F16"])
        step = 256 if w == "Q4_K" else 32
        dtype = rng.choice(["F16", "F16", "BF16"]) if w != "F16" else "F16"
        rows = rng.choice([1, _log(rng, 2, 24), _log(rng, 25, 600), _log(rng, 600, 3500)])
        if dtype == "BF16":
            rows = max(rows, 25)
        d = _multiple(_log(rng, 384, 3072), step)
        act = rng.choice(["gelu", "silu_gate"])
        ff = _multiple(d * rng.uniform(2.5, 4), step)
        return {"kind": "mlp", "weights": w, "act": act, "dtype": dtype, "blocks": rng.randint(1, 6) if rows < 600 else 1, "d": d, "ff": ff,
                "batch": 1, "rows": rows, "bias": act == "gelu"}
    if kind == "linear":
        d = _multiple(_log(rng, 384, 3072), 4)
        return {"kind": "linear", "d": d, "out": int(d * rng.uniform(1, 4)), "rows": _log(rng, 16, 512)}
    rows = rng.choice([1, _log(rng, 16, 1500)])
    return {"kind": "attention", "heads": rng.choice([6, 16, 32]), "dim": rng.choice([64, 72, 80, 96]), "rows": rows,
            "context": _log(rng, 100, 2000) if rows == 1 else rows, "scores": rng.choice(["F32", "F16"])}


# ------------------------------------------------------------------------------------------------ tensors on the device

class _Memory:
    """A library buffer as torch sees it; holds the buffer."""

    def __init__(self, tensor, nbytes):
        self.tensor = tensor
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (tensor.ptr, False), "version": 2}


def _view(t):
    """The values of a plain device tensor, in place."""
    raw = torch.as_tensor(_Memory(t, t.numel() * t.dt.size_of()), device="cuda")
    return raw.view(TORCH[t.dt.name]).view(t.shape)


def _to_device(gpu, values, dt):
    """A device tensor that holds `values` (a torch tensor, or a list of byte tensors with their offsets)."""
    shape = list(values.shape) if isinstance(values, torch.Tensor) else values[0]
    numel = math.prod(shape)
    t = Tensor(shape, dt, gpu, GpuBuffer(gpu, dt.nbytes(numel)))
    if isinstance(values, torch.Tensor):
        values = (shape, [(0, values.contiguous().view(torch.uint8).reshape(-1))])
    raw = torch.as_tensor(_Memory(t, dt.nbytes(numel)), device="cuda")
    for offset, part in values[1]:
        raw[offset:offset + part.numel()].copy_(part)
    return t


def quantise_q8(w, dt):
    """Blocks of 32: d = amax / 127, codes round(w / d); codes and scales in the format's two segments."""
    b = w.reshape(-1, 32)
    d = b.abs().amax(1, keepdim=True) / 127
    q = torch.where(d > 0, torch.round(b / d), 0).to(torch.int8)
    scales = d.to(torch.float16 if dt == DType.Q8_0H else torch.float32)
    return list(w.shape), [(dt.segments(w.numel())[0][0], q.view(torch.uint8).reshape(-1)),
                           (dt.segments(w.numel())[1][0], scales.view(torch.uint8).reshape(-1))]


def quantise_q4k(w):
    """Super-blocks of 256: eight sub-blocks of 32 with 6-bit scales and minima under an f16 d and dmin, 4-bit codes."""
    b = w.reshape(-1, 8, 32)
    low = (-b.amin(2)).clamp_min(0)
    step = (b.amax(2) + low) / 15
    d = (step.amax(1, keepdim=True) / 63).to(torch.float16)
    dmin = (low.amax(1, keepdim=True) / 63).to(torch.float16)
    ratio = lambda v, s: torch.where(s > 0, torch.round(v / s.float()), 0).clamp(0, 63)  # noqa: E731
    sc, mn = ratio(step, d), ratio(low, dmin)
    scale, shift = (sc * d.float())[..., None], (mn * dmin.float())[..., None]
    q = torch.where(scale > 0, torch.round((b + shift) / scale), 0).clamp(0, 15).to(torch.uint8)
    sc, mn = sc.to(torch.uint8), mn.to(torch.uint8)
    head = torch.cat([d.view(torch.uint8), dmin.view(torch.uint8),
                      sc[:, :4] | (sc[:, 4:] >> 4 << 6), mn[:, :4] | (mn[:, 4:] >> 4 << 6), (sc[:, 4:] & 15) | (mn[:, 4:] & 15) << 4], 1)
    codes = (q[:, 0::2] | q[:, 1::2] << 4).reshape(-1, 128)
    return list(w.shape), [(0, torch.cat([head, codes], 1).reshape(-1))]


def _weight(gpu, gen, rows, k, dt, gain=1.0):
    w = torch.randn((rows, k), generator=gen, device="cuda") * (gain / math.sqrt(k))
    if dt in (DType.Q8_0H, DType.Q8_0F):
        return _to_device(gpu, quantise_q8(w, dt), dt)
    if dt == DType.Q4_K:
        return _to_device(gpu, quantise_q4k(w), dt)
    return _to_device(gpu, w.to(TORCH[dt.name]), dt)


def _normal(gpu, gen, shape, name, std=1.0):
    return _to_device(gpu, (torch.randn(shape, generator=gen, device="cuda") * std).to(TORCH[name]), DType[name])


#: keeps a token's scale through fc1, GELU and fc2: 1 / rms(gelu(N(0, 1)))
AFTER_GELU = 1.534


# ------------------------------------------------------------------------------------------------ prepare and run

def prepare(case, seed):
    torch.cuda.synchronize()  # memory that earlier states gave back is free of work
    gpu = Device.request_device(DeviceRequest.GPU, 0)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = types.SimpleNamespace(kind=case["kind"])
    {"lazy": _prepare_lazy, "decode": _prepare_decode, "mlp": _prepare_mlp, "linear": _prepare_linear,
     "attention": _prepare_attention}[s.kind](s, case, gpu, gen)
    torch.cuda.synchronize()
    return s


def _prepare_lazy(s, c, gpu, gen):
    dt, d, ff = DType[c["weights"]], c["d"], c["ff"]
    s.linears = []
    for _ in range(c["layers"]):
        s.linears += [Linear(_weight(gpu, gen, d, d, dt), _normal(gpu, gen, (d,), "F16", 0.02)),
                      Linear(_weight(gpu, gen, ff, d, dt), _normal(gpu, gen, (ff,), "F16", 0.02), rb.EPILOGUE_GELU_TANH),
                      Linear(_weight(gpu, gen, d, ff, dt, AFTER_GELU), _normal(gpu, gen, (d,), "F16", 0.02))]
    s.linears.append(Linear(_weight(gpu, gen, c["vocab"], d, dt), _normal(gpu, gen, (c["vocab"],), "F16", 0.02)))
    s.x = _normal(gpu, gen, (1, c["rows"], d), "F16")


def _prepare_decode(s, c, gpu, gen):
    dt, name, d, ff = DType[c["weights"]], "F32" if c["weights"] == "Q8_0F" else "F16", c["d"], c["ff"]
    s.x = h = _normal(gpu, gen, (1, 1, d), name)
    nodes = []
    for _ in range(c["layers"]):
        fc1 = Linear(_weight(gpu, gen, ff, d, dt), _normal(gpu, gen, (ff,), name, 0.02), rb.EPILOGUE_GELU_TANH)
        fc2 = Linear(_weight(gpu, gen, d, ff, dt, AFTER_GELU), _normal(gpu, gen, (d,), name, 0.02))
        nodes += [fc1.schedule(h)]
        nodes += [fc2.schedule(nodes[-1])]
        h = nodes[-1]
    torch.cuda.synchronize()
    h.resolve()
    s.exe = Executable(gpu, nodes)
    s.out = _view(h)


def _prepare_mlp(s, c, gpu, gen):
    dt, name, d, ff = DType[c["weights"]], c["dtype"], c["d"], c["ff"]
    wide = 2 * ff if c["act"] == "silu_gate" else ff
    bias = lambda n: _normal(gpu, gen, (n,), name, 0.02) if c["bias"] else None  # noqa: E731
    s.blocks, s.out = [], []
    for _ in range(c["blocks"]):
        mlp = MLP(Linear(_weight(gpu, gen, wide, d, dt), bias(wide)), Linear(_weight(gpu, gen, d, ff, dt, AFTER_GELU), bias(d)), act=c["act"])
        x = _normal(gpu, gen, (c["batch"], c["rows"], d), name)
        torch.cuda.synchronize()
        s.blocks.append((mlp, x))
        s.out.append(_view(mlp.bind(x)[1]))


def _prepare_linear(s, c, gpu, gen):
    lin = Linear(_weight(gpu, gen, c["out"], c["d"], DType.F32), _normal(gpu, gen, (c["out"],), "F32", 0.02))
    s.x = _normal(gpu, gen, (1, c["rows"], c["d"]), "F32")
    torch.cuda.synchronize()
    y = lin.schedule(s.x).resolve()
    s.exe, s.out = Executable(gpu, [y]), _view(y)


def _prepare_attention(s, c, gpu, gen):
    h, rows, t, dim = c["heads"], c["rows"], c["context"], c["dim"]
    q, k = _normal(gpu, gen, (1, h, rows, dim), c["scores"], 1 / math.sqrt(dim)), _normal(gpu, gen, (1, h, dim, t), c["scores"])
    p = _to_device(gpu, torch.softmax(torch.randn((1, h, rows, t), generator=gen, device="cuda"), -1).half(), DType.F16)
    v = _normal(gpu, gen, (1, h, t, dim), "F16")
    torch.cuda.synchronize()
    scores, values = q.matmul(k).resolve(), p.matmul(v).resolve()
    s.exe, s.out, s.keep = Executable(gpu, [scores, values]), [_view(scores), _view(values)], (q, k, p, v)


def run(s):
    if s.kind == "lazy":
        h = s.x
        for lin in s.linears:
            h = lin.schedule(h)
        return h.resolve().to(Device.CPU).to_numpy()
    if s.kind == "mlp":
        for mlp, x in s.blocks:
            mlp.schedule(x)
        return s.out
    s.exe.dispatch()
    return s.out


# ------------------------------------------------------------------------------------------------ work and tolerance

def _linear_work(rows, n, k, weights, activations, bias):
    """(bytes of weights and bias, flops) of a Linear."""
    return n * k * BYTES[weights] + (n * BYTES[activations] if bias else 0), 2.0 * rows * n * k


def work(case):
    """The weights, and the activations that enter and leave the pass (what one node hands to the next is not counted)."""
    c, kind = case, case["kind"]
    if kind == "lazy":
        d, ff, m, w = c["d"], c["ff"], c["rows"], c["weights"]
        nodes = [_linear_work(m, n, k, w, "F16", True) for n, k in [(d, d), (ff, d), (d, ff)] * c["layers"] + [(c["vocab"], d)]]
        ends = m * (d + c["vocab"]) * 2
    elif kind == "decode":
        d, ff, w, a = c["d"], c["ff"], c["weights"], "F32" if c["weights"] == "Q8_0F" else "F16"
        nodes = [_linear_work(1, n, k, w, a, True) for n, k in [(ff, d), (d, ff)] * c["layers"]]
        ends = 2 * d * BYTES[a]
    elif kind == "mlp":
        d, ff, m = c["d"], c["ff"], c["batch"] * c["rows"]
        wide = 2 * ff if c["act"] == "silu_gate" else ff
        nodes = [_linear_work(m, n, k, c["weights"], c["dtype"], c["bias"]) for n, k in [(wide, d), (d, ff)] * c["blocks"]]
        ends = c["blocks"] * 2 * m * d * BYTES[c["dtype"]]
    elif kind == "linear":
        nodes = [_linear_work(c["rows"], c["out"], c["d"], "F32", "F32", True)]
        ends = c["rows"] * (c["d"] + c["out"]) * 4
    else:
        h, m, t, dim = c["heads"], c["rows"], c["context"], c["dim"]
        ends = h * ((m * dim + dim * t + m * t) * BYTES[c["scores"]] + (m * t + t * dim + m * dim) * 2)
        nodes = [(0, 4.0 * h * m * t * dim)]
    return {"bytes": sum(n[0] for n in nodes) + ends, "flops": sum(n[1] for n in nodes)}


def tolerance(case):
    """Two correct implementations round the same sums: 2^-11 (f16) or 2^-8 (bf16) of a value at most, once per tensor of
    the pass; a chain feeds each node's rounding to the next, and independent errors add as their squares."""
    kind = case["kind"]
    f32 = kind == "linear" or (kind == "decode" and case["weights"] == "Q8_0F")
    if f32:
        return {"rel": 1e-5}
    if kind == "mlp" and case["dtype"] == "BF16":
        return {"rel": 1e-2}
    nodes = {"lazy": 3 * case.get("layers", 0) + 1, "decode": 2 * case.get("layers", 0)}.get(kind, 2)
    return {"rel": 1e-3 * max(1.0, math.sqrt(nodes))}
