"""The work that users of this library have it do, as cases that can be timed and compared.

    listed()          the cases themselves
    draw(rng)         one more case from the same ranges
    prepare(case, s)  what a program has in hand before the call, on the GPU, made from seed s
    run(state)        one pass through the public entry points; returns its outputs
    work(case)        bytes and flops one pass cannot do without
    tolerance(case)   how far another correct implementation may be off
    exact(case, s)    the same outputs in plain torch and 64 bits

Five kinds of work, each through the entry point a program calls:

    matvec     yvex_b200_gemv            one encoded matrix times one or a few f32 rows
    batch      yvex_b200_gemv_batch      many encoded matrices of one shape, one input row each
    decode     yvex_b200_moe_decode      an MoE FFN layer at decode width, rows resident
    table      execute_rows              the same layer through the C11 operation table: host rows in and out, four residual
                                         streams (mHC envelope), resident weights named by host pointers
    prefill    yvex_b200_moe_wide        the MoE FFN layer over a prompt
    attention  yvex_b200_attention_gqa_decode   one position per session against a bf16 KV cache

Weights are random GGUF blocks (every payload pattern is a valid code, block scales uniform in [1e-4, 1e-3]), activations and
router logits N(0, 1), router weights N(0, 0.02): the distributions of the benchmark's configurations.
"""
from __future__ import annotations

import ctypes as C
import re
from pathlib import Path

import numpy as np
import torch

from yvex_b200 import lib, synth
from yvex_b200.workloads import device_blocks

QTYPES = {"IQ2_XXS": synth.IQ2_XXS, "Q2_K": synth.Q2_K, "Q4_K": synth.Q4_K, "Q8_0": synth.Q8_0, "MXFP4": synth.MXFP4,
          "BF16": synth.BF16, "F16": synth.F16, "F32": synth.F32}
BLOCK = ("IQ2_XXS", "Q2_K", "Q4_K", "Q8_0", "MXFP4")
GIB = 1 << 30


def _layer(hidden, experts, topk, inter, gate, down):
    return dict(hidden=hidden, experts=experts, topk=topk, inter=inter, gate=gate, down=down)


# The two layer shapes of the benchmark: a DeepSeek-style layer of 64 experts, and the large one of 256.
SMALL = _layer(4096, 64, 6, 1536, "IQ2_XXS", "Q4_K")
LARGE = _layer(7168, 256, 8, 2048, "IQ2_XXS", "Q4_K")


def listed():
    return [
        # One projection of one token: the smallest call, all latency.
        dict(name="matvec_iq2", kind="matvec", qtype="IQ2_XXS", rows=4096, width=4096, inputs=1),
        # A projection for the eight rows of a verification or micro-batch step.
        dict(name="matvec_q8_8rows", kind="matvec", qtype="Q8_0", rows=4096, width=4096, inputs=8),
        # The output head: one vocabulary-sized BF16 matrix per generated token.
        dict(name="matvec_head", kind="matvec", qtype="BF16", rows=129280, width=4096, inputs=1),
        # A stack of equal projections in one call: the matvec at streaming size.
        dict(name="batch_iq2", kind="batch", qtype="IQ2_XXS", rows=4096, width=4096, count=256),
        # One generated token through one layer.
        dict(name="decode_1", kind="decode", tokens=1, router="weights", **SMALL),
        # A serving step: a ragged batch of sessions, one token each, through the large layer.
        dict(name="decode_13_large", kind="decode", tokens=13, router="weights", **LARGE),
        # A token through the operation table as a runtime drives it: envelope, host rows, Q2_K down (the reference's own pair).
        dict(name="table_1", kind="table", tokens=1, streams=4, router="weights", **dict(SMALL, down="Q2_K")),
        # A short prompt, ragged against every tile size.
        dict(name="prefill_333", kind="prefill", tokens=333, router="weights", **dict(SMALL, down="Q2_K")),
        # An ordinary prompt.
        dict(name="prefill_2048", kind="prefill", tokens=2048, router="logits", **SMALL),
        # The largest: a long prompt, or many, through the large layer.
        dict(name="prefill_16384", kind="prefill", tokens=16384, router="logits", **LARGE),
        # Attention of a short conversation: one session, latency.
        dict(name="attention_short", kind="attention", sessions=1, q_heads=32, kv_heads=8, dim=128, visible=1500, context=4096),
        # Attention of a serving step at full context.
        dict(name="attention_long", kind="attention", sessions=16, q_heads=32, kv_heads=8, dim=128, visible=32768, context=32768),
    ]


# ---- sizes ------------------------------------------------------------------------------------------------------------

def _log(rng, lo, hi, step=1):
    """A size spread evenly over the logarithm of [lo, hi], a multiple of step."""
    v = lo * (hi / lo) ** rng.random()
    return int(min(hi, max(lo, round(v / step) * step)))


def _row_bytes(name, width):
    return synth.row_bytes(QTYPES[name], width)


def _expert_bytes(c):
    return 2 * c["inter"] * _row_bytes(c["gate"], c["hidden"]) + c["hidden"] * _row_bytes(c["down"], c["inter"])


def _draw_layer(rng, block, most_bytes):
    while True:
        c = _layer(_log(rng, 1024, 7168, 256), rng.choice((16, 32, 64, 96, 128, 160, 256)), rng.randint(1, 8),
                   _log(rng, 512, 2048, 256), rng.choice(("IQ2_XXS",) * 3 + block), rng.choice(block))
        if "MXFP4" in (c["gate"], c["down"]) and (c["hidden"] % 512 or c["inter"] % 512):
            continue                                                   # rows of MXFP4 experts come in pairs of 256 weights
        if (c["experts"] + 1) * _expert_bytes(c) <= most_bytes:
            return c


def draw(rng):
    kind = rng.choice(("matvec", "matvec", "batch", "decode", "decode", "table", "prefill", "prefill", "prefill", "attention", "attention"))
    if kind == "matvec":
        q = rng.choice(tuple(QTYPES))
        while True:
            rows, width, inputs = _log(rng, 256, 131072), _log(rng, 256, 8192, 256), rng.choice((1, 1, 1, _log(rng, 2, 16)))
            if q == "MXFP4" and width % 512:
                continue
            if rows * _row_bytes(q, width) <= 1.1 * GIB and rows * width * inputs <= 2 * 129280 * 4096:
                return dict(kind=kind, qtype=q, rows=rows, width=width, inputs=inputs)
    if kind == "batch":
        q = rng.choice(BLOCK)
        while True:
            rows, width, count = _log(rng, 256, 8192), _log(rng, 512, 8192, 512), _log(rng, 2, 256)
            rows -= rows % 8                                           # every matrix of the stack starts on a 16-byte boundary
            if count * rows * _row_bytes(q, width) <= 1.1 * GIB:
                return dict(kind=kind, qtype=q, rows=rows, width=width, count=count)
    if kind == "decode":
        return dict(kind=kind, tokens=_log(rng, 1, 62), router=rng.choice(("weights", "weights", "logits")), **_draw_layer(rng, BLOCK, 3 * GIB))
    if kind == "table":
        return dict(kind=kind, tokens=_log(rng, 1, 62), streams=rng.choice((1, 4)), router="weights",
                    **_draw_layer(rng, ("Q2_K", "Q4_K"), GIB // 2))
    if kind == "prefill":
        while True:
            c = dict(kind=kind, tokens=_log(rng, 64, 16384), router=rng.choice(("weights", "logits")),
                     **_draw_layer(rng, ("IQ2_XXS", "Q2_K", "Q4_K"), 4 * GIB))
            # affine gate and up projections cost more per product than IQ2_XXS, and the router's projection counts too
            cost = c["tokens"] * ((c["topk"] + 1) * 6.0 * c["hidden"] * c["inter"] * (2.0 if c["gate"] != "IQ2_XXS" else 1.0) +
                                  (60.0 * c["hidden"] * c["experts"] if c["router"] == "weights" else 0.0))
            if cost <= 0.8 * 16384 * 9 * 6.0 * 7168 * 2048:
                return c
    while True:
        kv, dim = rng.choice((1, 2, 4, 8, 16)), rng.choice((64, 128, 128, 256))
        c = dict(kind=kind, sessions=_log(rng, 1, 64), q_heads=kv * rng.choice((1, 2, 4)), kv_heads=kv, dim=dim,
                 visible=_log(rng, 100, 131072))
        c["context"] = c["visible"] + rng.choice((0, _log(rng, 1, 4096)))
        if c["sessions"] * kv * c["context"] * dim * 4 <= 2 * GIB:
            return c


# ---- inputs -----------------------------------------------------------------------------------------------------------

def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed & 0x7fffffff)
    return gen


def _matrix(name, rows, width, gen):
    """`rows` encoded rows of `width` weights as device bytes."""
    if name in BLOCK:
        return device_blocks(torch, QTYPES[name], rows, width, gen, "cuda")
    w = torch.randn((rows, width), device="cuda", generator=gen) * 0.02
    return w.to({"BF16": torch.bfloat16, "F16": torch.float16, "F32": torch.float32}[name]).view(torch.uint8).reshape(-1)


def _spec(c):
    return synth.MoELayerSpec(c["hidden"], c["experts"], c["topk"], c["inter"], gate_qtype=QTYPES[c["gate"]], down_qtype=QTYPES[c["down"]])


def _experts(c, gen):
    H, I, E = c["hidden"], c["inter"], c["experts"]
    t = dict(gate=_matrix(c["gate"], E * I, H, gen), up=_matrix(c["gate"], E * I, H, gen), down=_matrix(c["down"], E * H, I, gen),
             shared_gate=_matrix(c["gate"], I, H, gen), shared_up=_matrix(c["gate"], I, H, gen), shared_down=_matrix(c["down"], H, I, gen))
    if c["router"] == "weights":
        t["router"] = torch.randn((E, H), device="cuda", generator=gen) * 0.02
    return t


def _table_inputs(c, gen):
    """The resident arrays of one layer (with its envelope when there are several streams) and the input rows."""
    t, S, H = _experts(c, gen), c["streams"], c["hidden"]
    randn = lambda *shape: torch.randn(shape, device="cuda", generator=gen)  # noqa: E731
    if S > 1:
        t["mhc_fn"] = randn((S + 2) * S, S * H) * 0.05
        t["mhc_scale"] = torch.tensor([0.7, 1.3, 0.9], device="cuda")
        t["mhc_base"] = randn((S + 2) * S) * 0.3
        t["ffn_norm"] = 1.0 + 0.1 * randn(H)
    return t, randn(c["tokens"], S * H)


class _Table:
    """A backend session as a runtime holds it: resident arena, attached workspace, one layer job, page-locked host rows."""

    def __init__(self, c, gen):
        from yvex_b200 import backend as B
        self.B, T, H, S, k = B, c["tokens"], c["hidden"], c["streams"], c["topk"]
        tensors, rows = _table_inputs(c, gen)
        arrays = {n: v.cpu().numpy() for n, v in tensors.items()}
        self.rows_in = torch.empty((T, S * H), dtype=torch.float32).pin_memory()
        self.rows_in.copy_(rows)
        self.rows_out = torch.empty((T, S * H), dtype=torch.float32).pin_memory()
        self.selected, self.weights = np.zeros((T, k), np.uint64), np.zeros((T, k), np.float32)
        self.be = B.Backend()
        if self.be.rc != B.OK:
            raise RuntimeError(self.be.message())
        self.arena = B.ResidentArena(self.be, arrays)
        self.job = B.moe_job(self.arena, _spec(c), residual_streams=S)
        self.ops, need = B.moe_ops(self.be), B.ull()
        self._ok(self.ops.workspace_required(self.job.layer, T, C.byref(need), C.byref(self.be.err)))
        rc, ws, _ = self.be.tensor(need.value)
        self._ok(rc)
        self._ok(B._lib.yvex_backend_workspace_attach(self.be.h, ws, C.byref(self.be.err)))
        self.batch = B.row_batch(T, S * H, host_rows=self.rows_in.data_ptr())
        self.output = B.row_output(self.rows_out.data_ptr(), T * S * H, self.selected.ctypes.data, self.weights.ctypes.data, T * k)
        self.result = B.RowBatchResult()

    def _ok(self, rc):
        if rc != self.B.OK:
            raise RuntimeError(self.be.message())

    def execute(self):
        B = self.B
        self._ok(self.ops.execute_rows(self.be.h, C.byref(self.job), C.byref(self.batch), C.byref(self.output), C.byref(self.result),
                                       C.byref(self.be.err)))
        return dict(rows=self.rows_out, selected=self.selected, weights=self.weights)

    def __del__(self):
        if getattr(self, "be", None) is not None:
            self.arena = None
            self.be.close()


def prepare(case, seed):
    c, gen = case, _generator(seed)
    randn = lambda *shape: torch.randn(shape, device="cuda", generator=gen)  # noqa: E731
    s = dict(case=c, status=lib.Status())
    if c["kind"] == "matvec":
        s["weights"] = _matrix(c["qtype"], c["rows"], c["width"], gen)
        s["x"] = randn(c["inputs"], c["width"])
        s["out"] = torch.empty((c["inputs"], c["rows"]), device="cuda")
    elif c["kind"] == "batch":
        s["weights"] = _matrix(c["qtype"], c["count"] * c["rows"], c["width"], gen)
        s["x"] = randn(c["count"], c["width"])
        s["out"] = torch.empty((c["count"], c["rows"]), device="cuda")
    elif c["kind"] == "table":
        s["table"] = _Table(c, gen)
    elif c["kind"] == "attention":
        S, D = c["sessions"], c["dim"]
        s["q"] = randn(S, c["q_heads"], D).to(torch.bfloat16)
        s["k"], s["v"] = (torch.empty((S, c["kv_heads"], c["context"], D), dtype=torch.bfloat16, device="cuda").normal_(generator=gen)
                          for _ in range(2))
        s["out"] = torch.empty((S, c["q_heads"], D), device="cuda")
        s["workspace"] = torch.empty(max(256, int(lib.lib.yvex_b200_attention_workspace_bytes(S, c["q_heads"], c["kv_heads"], D, c["context"]))),
                                     dtype=torch.uint8, device="cuda")
    else:
        wide, T = c["kind"] == "prefill", c["tokens"]
        s["geometry"] = lib.geometry_of(_spec(c))
        s["weights"] = lib.weights_of(_experts(c, gen))
        s["x"] = randn(T, c["hidden"])
        s["logits"] = randn(T, c["experts"]) if c["router"] == "logits" else None
        s["workspace"] = torch.empty(lib.moe_workspace_bytes(s["geometry"], T, wide), dtype=torch.uint8, device="cuda")
        s["out"] = torch.empty_like(s["x"])
        s["selected"] = torch.empty((T, c["topk"]), dtype=torch.int32, device="cuda")
        s["route_weights"] = torch.empty((T, c["topk"]), device="cuda")
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "matvec":
        return lib.gemv(QTYPES[c["qtype"]], s["weights"], c["rows"], c["width"], s["x"], s["status"], out=s["out"])
    if c["kind"] == "batch":
        return lib.gemv_batch(QTYPES[c["qtype"]], s["weights"], c["count"], c["rows"], c["width"], s["x"], s["status"], out=s["out"])
    if c["kind"] == "table":
        return s["table"].execute()
    if c["kind"] == "attention":
        return lib.attention_gqa_decode(s["q"], s["k"], s["v"], c["visible"] - 1, c["dim"] ** -0.5, s["status"], workspace=s["workspace"],
                                        out=s["out"])
    return lib.moe_layer(s["geometry"], s["weights"], s["x"], s["status"], logits=s["logits"], wide=c["kind"] == "prefill",
                         workspace=s["workspace"], out=s["out"], selected=s["selected"], wts=s["route_weights"])


# ---- what a pass cannot do without --------------------------------------------------------------------------------------

def work(case):
    c = case
    if c["kind"] == "matvec":
        n = c["rows"] * c["width"]
        return dict(bytes=c["rows"] * _row_bytes(c["qtype"], c["width"]) + 4 * c["inputs"] * (c["rows"] + c["width"]), flops=2.0 * n * c["inputs"])
    if c["kind"] == "batch":
        return dict(bytes=c["count"] * (c["rows"] * _row_bytes(c["qtype"], c["width"]) + 4 * (c["rows"] + c["width"])),
                    flops=2.0 * c["count"] * c["rows"] * c["width"])
    if c["kind"] == "attention":
        kv, q = c["sessions"] * c["kv_heads"] * c["visible"] * c["dim"], c["sessions"] * c["q_heads"] * c["dim"]
        return dict(bytes=4 * kv + 6 * q, flops=4.0 * q * c["visible"])
    T, E, k, H = c["tokens"], c["experts"], c["topk"], c["hidden"]
    touched = E * (1.0 - (1.0 - k / E) ** T) + 1.0                     # experts that some token picks, and the shared one
    bytes_ = touched * _expert_bytes(c) + 8 * T * H * c.get("streams", 1) + 4 * E * (H if c["router"] == "weights" else T)
    flops = T * (k + 1) * 6.0 * H * c["inter"] + (2.0 * T * E * H if c["router"] == "weights" else 0.0)
    if c.get("streams", 1) > 1:
        mix = (c["streams"] + 2) * c["streams"] * c["streams"] * H
        bytes_, flops = bytes_ + 4 * mix, flops + 2.0 * T * mix
    return dict(bytes=bytes_, flops=flops)


def tolerance(case):
    """About four times what was measured: matvecs and attention against the same contraction in 64 bits over the decoded
    weights (at most 2.2e-7 and 1.9e-6, largest single values 1e-6 and 7.5e-6), a layer's decode path against its prefill path,
    whose sums run in another order (at most 2.5e-4 and 1.1e-2: the outputs are bf16 values of sums of bf16 values, and a few of
    them fall to the next one)."""
    if case["kind"] in ("matvec", "batch"):
        return {"rel": 1e-6, "max": 5e-6}
    if case["kind"] == "attention":
        return {"rel": 8e-6, "max": 4e-5}
    return {"rel": 1e-3, "max": 0.05}


# ---- the same outputs in 64 bits ------------------------------------------------------------------------------------------
# Plain torch over the block layouts of the GGUF format; sums and products in 64 bits, rounded where the layer is specified
# to round (bf16 of the ingress rows, of the SwiGLU products, of each expert's result and of the layer's; f32 of a projection).

def _codebook():
    """The IQ2_XXS magnitudes [256, 8], from the table of nibbles (digit 0, 1, 2 = 8, 25, 43) that the format fixes."""
    text = (Path(__file__).resolve().parent.parent / "yvex_b200" / "csrc" / "iq2xxs_grid_nibbles.inc").read_text()
    words = [int(v, 16) for v in re.findall(r"0x([0-9a-f]{8})u", text)]
    digits = torch.tensor([[(w >> (4 * i)) & 3 for i in range(8)] for w in words], device="cuda")
    return torch.tensor([8.0, 25.0, 43.0], dtype=torch.float64, device="cuda")[digits]


def _f16(b):
    return b.contiguous().view(torch.float16).double()


def _decoded(name, raw, rows, width):
    """Encoded rows as [rows, width] in 64 bits."""
    raw = raw.reshape(rows, -1)
    if name in ("F32", "F16", "BF16"):
        return raw.view({"F32": torch.float32, "F16": torch.float16, "BF16": torch.bfloat16}[name]).double()
    b = raw.reshape(-1, {"IQ2_XXS": 66, "Q2_K": 84, "Q4_K": 144, "Q8_0": 34, "MXFP4": 17}[name])
    if name == "Q8_0":
        w = _f16(b[:, :2]) * b[:, 2:].contiguous().view(torch.int8).double()
    elif name == "MXFP4":
        levels = torch.tensor([0, 1, 2, 3, 4, 6, 8, 12, 0, -1, -2, -3, -4, -6, -8, -12], dtype=torch.float64, device=b.device)
        codes = torch.cat((b[:, 1:] & 15, b[:, 1:] >> 4), 1).long()
        w = levels[codes] * torch.exp2(b[:, :1].double() - 128.0)
    elif name == "IQ2_XXS":
        groups = b[:, 2:].reshape(-1, 8, 8)
        bits = groups[:, :, 4:].contiguous().view(torch.int32).long().squeeze(-1) & 0xffffffff              # [n, 8]
        low = (bits[:, :, None] >> (7 * torch.arange(4, device=b.device))) & 127                            # [n, 8, 4]
        sign = (low[..., None] >> torch.arange(7, device=b.device)) & 1
        sign = torch.cat((sign, sign.sum(-1, keepdim=True) & 1), -1)                                        # the eighth makes the parity even
        scale = _f16(b[:, :2]) * 0.25 * (0.5 + (bits >> 28).double())                                       # [n, 8]
        w = scale[:, :, None, None] * _codebook()[groups[:, :, :4].long()] * (1.0 - 2.0 * sign)
    elif name == "Q2_K":
        planes = b[:, 16:80].reshape(-1, 2, 1, 32) >> (2 * torch.arange(4, device=b.device, dtype=torch.uint8))[:, None]
        code = (planes & 3).reshape(-1, 16, 16).double()
        w = _f16(b[:, 80:82])[..., None] * (b[:, :16] & 15).double()[..., None] * code - _f16(b[:, 82:])[..., None] * (b[:, :16] >> 4).double()[..., None]
    else:
        s = b[:, 4:16].long()
        scale = torch.cat((s[:, :4] & 63, (s[:, 8:] & 15) | (s[:, :4] >> 6 << 4)), 1).double()[..., None]
        least = torch.cat((s[:, 4:8] & 63, (s[:, 8:] >> 4) | (s[:, 4:8] >> 6 << 4)), 1).double()[..., None]
        q = b[:, 16:].reshape(-1, 4, 32)
        w = _f16(b[:, :2])[..., None] * scale * torch.stack((q & 15, q >> 4), 2).reshape(-1, 8, 32).double() - _f16(b[:, 2:4])[..., None] * least
    return w.reshape(rows, width)


def _bf16(v):
    return v.float().to(torch.bfloat16).double()


def _exact_layer(c, t, x, logits):
    """The layer on 64-bit rows: (result rows, selections, their weights)."""
    H, I, k = c["hidden"], c["inter"], c["topk"]
    spec = _spec(c)
    x = _bf16(x)
    logits = (x @ t["router"].double().T).float().double() if logits is None else logits.double()
    score = torch.nn.functional.softplus(logits, threshold=700.0).sqrt().float()
    selected = torch.sort(score, dim=1, descending=True, stable=True)[1][:, :k]
    weight = score.gather(1, selected).double()
    weight = weight / weight.sum(1, keepdim=True) * spec.scaling

    def expert(parts, rows, w):
        gate, up, down = (_decoded(c[q], p, n, m) for q, p, n, m in zip(("gate", "gate", "down"), parts, (I, I, H), (H, H, I)))
        g, u = (x[rows] @ gate.T).clamp(max=spec.limit), (x[rows] @ up.T).clamp(-spec.limit, spec.limit)
        return _bf16(_bf16(g * torch.sigmoid(g) * u * w[:, None]) @ down.T).float()

    every = torch.arange(x.shape[0], device=x.device)
    pairs = torch.zeros((x.shape[0], k, H), device=x.device)
    packs = [t[n].reshape(c["experts"], -1) for n in ("gate", "up", "down")]
    for e in selected.unique().tolist():
        row, rank = (selected == e).nonzero(as_tuple=True)
        pairs[row, rank] = expert([p[e] for p in packs], row, weight[row, rank])
    shared = expert([t["shared_gate"], t["shared_up"], t["shared_down"]], every, torch.ones_like(weight[:, 0]))
    out = shared.double()
    for r in range(k):
        out += pairs[:, r]
    return _bf16(out), selected, weight


def _exact_table(c, gen):
    t, rows = _table_inputs(c, gen)
    S, H, eps = c["streams"], c["hidden"], 1e-6
    x = rows.double()
    if S == 1:
        return _exact_layer(c, t, x, None)
    scale, base = t["mhc_scale"].double(), t["mhc_base"].double()
    mix = (x @ t["mhc_fn"].double().T) / (x.square().mean(1, keepdim=True) + eps).sqrt()
    pre = torch.sigmoid(mix[:, :S] * scale[0] + base[:S]) + eps
    post = 2.0 * torch.sigmoid(mix[:, S:2 * S] * scale[1] + base[S:2 * S])
    comb = torch.softmax((mix[:, 2 * S:] * scale[2] + base[2 * S:]).reshape(-1, S, S), 2) + eps
    for n in range(20):
        if n:
            comb = comb / (comb.sum(2, keepdim=True) + eps)
        comb = comb / (comb.sum(1, keepdim=True) + eps)
    streams = x.reshape(-1, S, H)
    flat = _bf16((pre[..., None] * streams).sum(1))
    normed = _bf16(flat / (flat.square().mean(1, keepdim=True) + eps).sqrt() * t["ffn_norm"].double())
    core, selected, weight = _exact_layer(c, t, normed, None)
    out = _bf16(post[..., None] * core[:, None] + torch.einsum("nst,nsh->nth", comb, streams))
    return out.reshape(-1, S * H), selected, weight


def exact(case, seed):
    c = case
    if c["kind"] == "matvec":
        s = prepare(c, seed)
        step = max(1, (1 << 27) // c["width"])                          # rows at a time: a decoded head is several GB
        cuts = [(a, min(a + step, c["rows"])) for a in range(0, c["rows"], step)]
        raw = s["weights"].reshape(c["rows"], -1)
        return torch.cat([s["x"].double() @ _decoded(c["qtype"], raw[a:b].contiguous(), b - a, c["width"]).T for a, b in cuts], 1)
    if c["kind"] == "batch":
        s = prepare(c, seed)
        raw = s["weights"].reshape(c["count"], -1)
        return torch.stack([_decoded(c["qtype"], raw[m], c["rows"], c["width"]) @ s["x"][m].double() for m in range(c["count"])])
    if c["kind"] == "table":
        out, selected, weight = _exact_table(c, _generator(seed))
        return dict(rows=out.cpu(), selected=selected.cpu().numpy().astype(np.uint64), weights=weight.cpu().numpy())
    if c["kind"] == "attention":
        s, V, group = prepare(c, seed), c["visible"], c["q_heads"] // c["kv_heads"]
        out = torch.empty((c["sessions"], c["q_heads"], c["dim"]), dtype=torch.float64, device="cuda")
        for n in range(c["sessions"]):
            for h in range(c["kv_heads"]):
                q = s["q"][n, h * group:(h + 1) * group].double()
                p = torch.softmax(q @ s["k"][n, h, :V].double().T * c["dim"] ** -0.5, 1)
                out[n, h * group:(h + 1) * group] = p @ s["v"][n, h, :V].double()
        return out
    gen = _generator(seed)
    t, T = _experts(c, gen), c["tokens"]
    x = torch.randn((T, c["hidden"]), device="cuda", generator=gen)
    logits = torch.randn((T, c["experts"]), device="cuda", generator=gen) if c["router"] == "logits" else None
    out, selected, weight = _exact_layer(c, t, x.double(), logits)
    return out, selected.int(), weight
