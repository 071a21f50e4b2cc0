"""The work a program hands to this library, as measurable cases.

A case is one pass over a set of weight tensors through vinf_3080ti_b200.runtime.Runtime:

  call       what is called                                                    stands for
  matvec     Runtime.matvec: host vector in, host vector out                   the synchronous single-row entry
  qmv        Runtime.qmv for every tensor of the list                          projections of a decode step, a verification
                                                                               pass, or (with `prompt`) a prompt pass
  layer      the seven matvecs of a decoder layer; `style` says whether as     the executor's layer, in its three spellings
             qmv, qmv_group (q/k/v and gate/up together) or qmv_fused (norm,
             silu * up and residual inside the matvecs)
  head       write + qmv_argmax                                                the LM head of a greedy step
  decode     write + one graph of `layers` layers and the LM head + ids        a whole decode pass

Weights are raw GGUF blocks with uniform-random quants and fp16 scales uniform in [1e-3, 1e-2), activations N(0, 1): the
recipe of the benchmark configurations.  Codebooks have random entries over the magnitudes of their formats.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vinf_3080ti_b200.gguf_types import CODEBOOK_BYTES, F16_FIELDS, TRAITS, GGUFTensorType
from vinf_3080ti_b200.runtime import Runtime

# The magnitudes that occur in each codebook.
CODEBOOK_VALUES = {
    "iq2xxs_grid": (8, 25, 43),
    "iq2xs_grid": (8, 25, 43),
    "iq2s_grid": (8, 25, 43),
    "iq3xxs_grid": (4, 12, 20, 28, 36, 44, 52, 62),
    "iq3s_grid": (1, 3, 5, 7, 9, 11, 13, 15),
}
PROMPT_ROWS = 64  # passes of this many rows or more are prompt passes (set_gemm_min_rows)
LAYER_27B = {"hidden": 5120, "ffn": 17408, "q": 6144, "kv": 1024}
IQ_SWEEP = "IQ2_XXS:17408x5120 IQ2_S:17408x5120 IQ3_S:17408x5120 IQ4_XS:17408x5120 IQ4_NL:5120x17408"


def listed():
    return [
        # One vector from the host through one small projection and back: call overhead, copies, one launch.
        {"name": "host_vector", "call": "matvec", "tensors": "Q6_K:1024x5120", "ntok": 1},
        # The few-row projections of a linear-attention layer (gates): a launch with almost nothing to read.
        {"name": "small_projections", "call": "qmv", "tensors": "Q8_0:48x5120 F32:48x5120", "ntok": 1},
        # The plain matvec of a decode step.
        {"name": "q4k_single", "call": "qmv", "tensors": "Q4_K:17408x5120", "ntok": 1},
        # A decoder layer, one token, the calls a drop-in executor makes.
        {"name": "layer_1", "call": "layer", "style": "qmv", "ntok": 1, **LAYER_27B},
        # The same layer for a 4-row verification pass, element-wise work inside the matvecs.
        {"name": "layer_4_fused", "call": "layer", "style": "fused", "ntok": 4, **LAYER_27B},
        # The widest small pass.
        {"name": "layer_8_group", "call": "layer", "style": "group", "ntok": 8, **LAYER_27B},
        # The codebook and non-linear types.
        {"name": "iq_sweep_1", "call": "qmv", "tensors": IQ_SWEEP, "ntok": 1},
        {"name": "iq_sweep_8", "call": "qmv", "tensors": IQ_SWEEP, "ntok": 8},
        # The remaining types at ragged sizes (rows that fill no tile evenly), a two-row pass.
        {"name": "other_types_2", "call": "qmv", "ntok": 2,
         "tensors": "Q8_0:4099x4096 Q5_K:11009x4096 Q2_K:9001x3584 F16:3073x4096 IQ2_XS:8191x5120 IQ3_XXS:6007x6144"},
        # The remainder of a prompt: more rows than a verification pass, fewer than a prompt pass.
        {"name": "short_prompt_24", "call": "qmv", "ntok": 24,
         "tensors": "Q6_K:6144x5120 Q3_K:17408x5120 Q4_K:5120x17408"},
        # A prompt pass over a layer's big tensors.
        {"name": "prompt_512", "call": "qmv", "prompt": True, "ntok": 512,
         "tensors": "Q6_K:6144x5120 Q3_K:17408x5120 Q4_K:17408x5120 Q4_K:5120x17408"},
        # A whole verification pass of the 27B model: 64 layers and the LM head, 12.6 GB of weights.
        {"name": "decode_pass_4", "call": "decode", "layers": 64, "vocab": 151936, "ntok": 4, **LAYER_27B},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tensor(rng, max_bytes):
    t = rng.choice([t for t in TRAITS])
    block, size = TRAITS[t]
    while True:
        rows = _log(rng, 16, 150000)
        cols = _log(rng, 256, 18432) // max(block, 32) * max(block, 32)
        if rows * (cols // block) * size <= max_bytes:
            return f"{t.name}:{rows}x{cols}"


def draw(rng):
    kind = rng.choice(["matvec", "qmv", "qmv", "qmv", "layer", "layer", "head", "prompt", "prompt", "short", "decode"])
    ntok = rng.randint(1, 8)
    if kind == "matvec":
        return {"call": "matvec", "tensors": _tensor(rng, 400e6), "ntok": 1}
    if kind == "qmv":
        return {"call": "qmv", "tensors": " ".join(_tensor(rng, 400e6) for _ in range(rng.randint(1, 3))), "ntok": ntok}
    if kind == "short":
        return {"call": "qmv", "tensors": _tensor(rng, 100e6), "ntok": rng.randint(9, 63)}
    if kind == "prompt":
        return {"call": "qmv", "prompt": True, "tensors": _tensor(rng, 100e6), "ntok": _log(rng, 64, 2048)}
    if kind == "head":
        return {"call": "head", "tensors": f"{rng.choice(['Q6_K', 'Q4_K', 'Q8_0', 'Q5_K'])}:{_log(rng, 32000, 152064)}x{256 * rng.randint(4, 24)}",
                "ntok": ntok}
    shape = {"hidden": 256 * _log(rng, 2, 24), "ffn": 256 * _log(rng, 4, 72), "q": 256 * _log(rng, 2, 24), "kv": 64 * _log(rng, 2, 24)}
    if kind == "layer":
        return {"call": "layer", "style": rng.choice(["qmv", "group", "fused"]), "ntok": ntok, **shape}
    return {"call": "decode", "layers": rng.randint(1, 12), "vocab": _log(rng, 8000, 152064), "ntok": ntok, **shape}


# ---- inputs ---------------------------------------------------------------------------------------------------------


def _parse(text):
    out = []
    for item in text.split():
        name, shape = item.split(":")
        rows, cols = shape.split("x")
        out.append((GGUFTensorType[name], int(rows), int(cols)))
    return out


def _layer_tensors(c):
    q6, q3, q4 = GGUFTensorType.Q6_K, GGUFTensorType.Q3_K, GGUFTensorType.Q4_K
    return [("q", q6, c["q"], c["hidden"]), ("k", q6, c["kv"], c["hidden"]), ("v", q6, c["kv"], c["hidden"]), ("o", q6, c["hidden"], c["q"]),
            ("gate", q3, c["ffn"], c["hidden"]), ("up", q3, c["ffn"], c["hidden"]), ("down", q4, c["hidden"], c["ffn"])]


def _nbytes(t, rows, cols):
    block, size = TRAITS[t]
    return rows * (cols // block) * size


def _blocks(t, rows, cols, gen):
    """Raw blocks of a tensor in device memory, readable a little past their end."""
    n = _nbytes(t, rows, cols)
    buf = torch.zeros((n + 16 + 255) // 256 * 256, dtype=torch.uint8, device="cuda")
    if t in (GGUFTensorType.F32, GGUFTensorType.F16):
        kind = torch.float32 if t is GGUFTensorType.F32 else torch.float16
        buf[:n].view(kind).uniform_(-1.0, 1.0, generator=gen)
        return buf
    buf[:n].random_(0, 256, generator=gen)
    size = TRAITS[t][1]
    raw = buf[:n].view(-1, size)
    for off in F16_FIELDS[t]:
        scale = torch.empty(raw.shape[0], dtype=torch.float32, device="cuda").uniform_(1e-3, 1e-2, generator=gen).half()
        raw[:, off:off + 2] = scale.view(torch.uint8).view(-1, 2)
    return buf


class _State:
    """A runtime with its tensors and buffers; what a program keeps between passes."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        rng = np.random.default_rng(seed)
        books = {n: rng.choice(np.array(CODEBOOK_VALUES[n], dtype=np.uint8), size=b).tobytes() for n, b in CODEBOOK_BYTES.items()}
        self.rt = Runtime(books["iq3s_grid"], codebooks=books)
        self.keep = {}

    def weight(self, name, t, rows, cols):
        self.keep["w." + name] = buf = _blocks(t, rows, cols, self.gen)
        self.rt.bind_tensor(name, buf.data_ptr(), int(t), cols, rows)

    def buffer(self, name, rows, cols, fill=None):
        self.keep[name] = buf = torch.zeros((rows, cols), dtype=torch.float32, device="cuda")
        if fill == "normal":
            buf.normal_(generator=self.gen)
        elif fill == "gain":
            buf.uniform_(0.5, 1.5, generator=self.gen)
        self.rt.bind(name, buf.data_ptr(), rows * cols)
        return buf

    def host(self, name, rows, cols):
        """Activations that a step brings from the host."""
        return torch.randn((rows, cols), generator=self.gen, device="cuda").cpu().numpy()


def prepare(case, seed):
    s = _State(seed)
    m, call = case["ntok"], case["call"]
    s.case = case
    if call in ("matvec", "qmv", "head"):
        s.tensors = _parse(case["tensors"])
        for i, (t, rows, cols) in enumerate(s.tensors):
            s.weight(f"w{i}", t, rows, cols)
            s.buffer(f"y{i}", m, rows)
            if f"x{cols}" not in s.keep:
                s.buffer(f"x{cols}", m, cols, "normal")
        s.x_host = s.host("x", m, s.tensors[0][2]) if call != "qmv" else None
        if case.get("prompt"):
            s.rt.set_gemm_min_rows(PROMPT_ROWS)
        return s
    layers = case.get("layers", 1)
    for n in range(layers):
        for name, t, rows, cols in _layer_tensors(case):
            s.weight(f"{n}.{name}", t, rows, cols)
            s.buffer(f"{n}.y.{name}", m, rows)
    s.buffer("x", m, case["hidden"], "normal")        # normalised hidden rows
    s.buffer("attn", m, case["q"], "normal")          # output of the attention itself
    s.buffer("act", m, case["ffn"], "normal")         # silu(gate) * up
    if case.get("style") == "fused":
        s.buffer("h0", m, case["hidden"], "normal")   # residual rows as the previous layer leaves them
        s.buffer("h", m, case["hidden"])
        s.buffer("norm1", 1, case["hidden"], "gain")
        s.buffer("norm2", 1, case["hidden"], "gain")
    if call == "decode":
        s.weight("head", GGUFTensorType.Q6_K, case["vocab"], case["hidden"])
        s.buffer("logits", m, case["vocab"])
        s.x_host = s.host("x", m, case["hidden"])
        torch.cuda.synchronize()
        s.rt.capture_begin()
        for n in range(layers):
            _layer_group(s.rt, n, m)
        s.rt.qmv_argmax("head", "x", "logits", m, blocking=False)
        s.graph = s.rt.capture_end()
    return s


# ---- passes ---------------------------------------------------------------------------------------------------------


def _layer_qmv(rt, n, m):
    rt.qmv(f"{n}.q", "x", f"{n}.y.q", m)
    rt.qmv(f"{n}.k", "x", f"{n}.y.k", m)
    rt.qmv(f"{n}.v", "x", f"{n}.y.v", m)
    rt.qmv(f"{n}.o", "attn", f"{n}.y.o", m)
    rt.qmv(f"{n}.gate", "x", f"{n}.y.gate", m)
    rt.qmv(f"{n}.up", "x", f"{n}.y.up", m)
    rt.qmv(f"{n}.down", "act", f"{n}.y.down", m)


def _layer_group(rt, n, m):
    rt.qmv_group([f"{n}.q", f"{n}.k", f"{n}.v"], "x", [f"{n}.y.q", f"{n}.y.k", f"{n}.y.v"], m)
    rt.qmv(f"{n}.o", "attn", f"{n}.y.o", m)
    rt.qmv_group([f"{n}.gate", f"{n}.up"], "x", [f"{n}.y.gate", f"{n}.y.up"], m)
    rt.qmv(f"{n}.down", "act", f"{n}.y.down", m)


def _layer_fused(rt, n, m, size):
    rt.copy("h", 0, "h0", 0, size)
    for name in ("q", "k", "v"):
        rt.qmv_fused(f"{n}.{name}", "h", f"{n}.y.{name}", m, norm="norm1")
    rt.qmv_fused(f"{n}.o", "attn", "h", m, add=True)
    for name in ("gate", "up"):
        rt.qmv_fused(f"{n}.{name}", "h", f"{n}.y.{name}", m, norm="norm2")
    rt.qmv_fused(f"{n}.down", f"{n}.y.gate", "h", m, silu_mul=f"{n}.y.up", add=True)


def run(s):
    case, rt = s.case, s.rt
    call, m = case["call"], case["ntok"]
    if call == "matvec":
        return [np.frombuffer(rt.matvec(f"w{i}", s.x_host), dtype=np.float32) for i in range(len(s.tensors))]
    if call == "qmv":
        for i, (_, _, cols) in enumerate(s.tensors):
            rt.qmv(f"w{i}", f"x{cols}", f"y{i}", m)
        return [s.keep[f"y{i}"] for i in range(len(s.tensors))]
    if call == "head":
        x = f"x{s.tensors[0][2]}"
        rt.write(x, s.x_host)
        ids = rt.qmv_argmax("w0", x, "y0", m)
        return {"ids": ids, "logits": s.keep["y0"]}
    if call == "decode":
        rt.write("x", s.x_host)
        rt.graph_launch(s.graph)
        ids = rt.argmax_fetch(m)
        last = case["layers"] - 1
        return {"ids": np.array(ids, dtype=np.int64), "logits": s.keep["logits"],
                "rows": [s.keep[f"{n}.y.{name}"] for n in sorted({0, last // 2, last}) for name in ("q", "k", "v", "o", "gate", "up", "down")]}
    if case["style"] == "fused":
        _layer_fused(rt, 0, m, m * case["hidden"])
        return {"h": s.keep["h"], "rows": [s.keep[f"0.y.{name}"] for name in ("q", "k", "v", "gate", "up")]}
    (_layer_qmv if case["style"] == "qmv" else _layer_group)(rt, 0, m)
    return [s.keep[f"0.y.{name}"] for name in ("q", "k", "v", "o", "gate", "up", "down")]


# ---- what a pass cannot do without, and how exact it is ---------------------------------------------------------------


def work(case):
    m = case["ntok"]
    if "tensors" in case:
        tensors = _parse(case["tensors"])
        inputs = sum({cols for _, _, cols in tensors})
    else:
        tensors = [(t, rows, cols) for _, t, rows, cols in _layer_tensors(case)] * case.get("layers", 1)
        inputs = case["hidden"] + case["q"] + case["ffn"]
        if case["call"] == "decode":
            tensors.append((GGUFTensorType.Q6_K, case["vocab"], case["hidden"]))
    weights = sum(_nbytes(t, rows, cols) for t, rows, cols in tensors)
    outputs = sum(rows for _, rows, _ in tensors)
    return {"bytes": weights + 4 * m * (inputs + outputs), "flops": 2 * m * sum(rows * cols for _, rows, cols in tensors)}


def tolerance(case):
    if case.get("prompt"):
        return {"rel": 1e-3}  # fp16 operands, 32-bit sums
    if case.get("style") == "fused":
        return {"rel": 2e-5}  # 32-bit sums through a norm, a second matvec, silu and a third
    return {"rel": 1e-5}  # 32-bit sums
