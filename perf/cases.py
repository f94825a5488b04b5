"""The work that a program built on this library has it do, as cases that can be timed and compared.

A case is a dict of plain values; `prepare` makes what such a program holds before the call (weights, scratch, input rows),
`run` is one pass through the public entry points. Kinds:

  decode   `tsp_moe_layer_decode` on 1..64 token rows: the generation step of a layer (a batch of one to a full batch), the
           verify pass of a few draft rows and the Q8_0 block of the draft model. `layers` consecutive layers with weights of
           their own make one pass, as a stack has them, so that small batches do not find their weights in L2.
  prefill  `tsp_moe_layer_prefill` on 65..4096 rows: a prompt or a chunk of one.
  head     the dense Q8_0 vocabulary matrix on 1..16 rows.
  top64    the sampler's top-64 rows of 1..16 rows of logits.
  edges    what surrounds the FFN in a layer: hyper-connection read, router projection (with the shared expert's gate row),
           hyper-connection write.

Weight forms: `q4_k` experts (Pack v3 planar or plain GGUF blocks), `q8_0` (the draft model's block, GGUF), `q5` (the model's
five-bit pairing: Q5_K gate / up, Q5_1 down, dense Q8_0 shared expert, GGUF). Layer shape where nothing else is said: 2048
channels, 512 experts of 512 hidden units, ten per token, one shared expert. Weights are N(0, 0.02) through the library's
encoders, activations N(0, 1), router logits N(0, 1), for prefill mostly with a Zipf(1.1) bias per expert.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from tokspur_public_b200 import capi, formats, synth
from tokspur_public_b200 import layer as L

CHANNELS, HIDDEN, EXPERTS, SELECTED = 2048, 512, 512, 10
VOCAB = 151936
BRANCHES = 4


def _layer(kind, tokens, weights, layout, dtype, layers=1, shared="same", skew=False, channels=CHANNELS, hidden=HIDDEN, experts=EXPERTS, selected=SELECTED):
    return {"kind": kind, "tokens": tokens, "weights": weights, "layout": layout, "dtype": dtype, "layers": layers, "shared": shared, "skew": skew,
            "channels": channels, "hidden": hidden, "experts": experts, "selected": selected}


def listed():
    def named(name, case):
        return dict(case, name=name)
    return [
        # one user generating: the smallest call there is, bound by launches and latency
        named("decode_1", _layer("decode", 1, "q4_k", "planar", "f16", layers=4)),
        # a small batch, or the verify pass of a few draft rows
        named("decode_8", _layer("decode", 8, "q4_k", "planar", "f16", layers=2)),
        # the full decode batch: most experts are hit once or twice
        named("decode_64", _layer("decode", 64, "q4_k", "planar", "f16")),
        # the draft model's block on the rows of one verify pass
        named("draft_block_5", _layer("decode", 5, "q8_0", "gguf", "f16")),
        # layers that the model keeps in its five-bit encodings, a ragged batch of FP32 rows as the C++ host layer passes them
        named("five_bit_13_f32", _layer("decode", 13, "q5", "gguf", "f32", layers=2, shared="q8_0")),
        # a long prompt (one full chunk), loads skewed over the experts
        named("prefill_4096", _layer("prefill", 4096, "q4_k", "planar", "f16", skew=True)),
        # a medium, ragged prompt in the model's mix of Q4_K experts and a dense Q8_0 shared expert, FP32 rows
        named("prefill_1003_mix_f32", _layer("prefill", 1003, "q4_k", "planar", "f32", shared="q8_0", skew=True)),
        # a short prompt
        named("prefill_160", _layer("prefill", 160, "q4_k", "planar", "f16", skew=True)),
        # the head behind a single generated row (an FP32 row out of the final norm), and behind a full verify pass
        {"name": "head_1", "kind": "head", "rows": 1, "vocabulary": VOCAB, "exact": False},
        {"name": "head_16", "kind": "head", "rows": 16, "vocabulary": VOCAB, "exact": True},
        # what the sampler reads of the verify pass's logits
        {"name": "top64_16", "kind": "top64", "rows": 16, "vocabulary": VOCAB},
        # the steps around the FFN for a chunk of a prompt
        {"name": "edges_2048", "kind": "edges", "tokens": 2048, "channels": CHANNELS, "experts": EXPERTS},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["decode"] * 4 + ["prefill"] * 4 + ["head", "head", "top64", "edges"])
    if kind == "head":
        return {"kind": "head", "rows": rng.randint(1, 16), "vocabulary": rng.choice([32000, 50304, 151936, 248320]), "exact": rng.random() < 0.5}
    if kind == "top64":
        return {"kind": "top64", "rows": rng.randint(1, 16), "vocabulary": rng.choice([32000, 50257, 151936, 248320])}
    if kind == "edges":
        return {"kind": "edges", "tokens": _log_int(rng, 1, 2048), "channels": rng.choice([1024, 2048, 2560]), "experts": rng.choice([64, 512])}
    shape = {}
    if rng.random() < 0.3:   # other layer shapes
        shape = {"channels": rng.choice([512, 1024, 2048]), "hidden": rng.choice([256, 512, 768]), "experts": rng.choice([16, 64, 128, 256]),
                 "selected": rng.choice([2, 4, 8])}
    dtype = rng.choice(["f16", "f32"])
    if kind == "prefill":
        tokens = _log_int(rng, 65, 4000)
        return _layer("prefill", tokens, "q4_k", rng.choice(["planar", "planar", "gguf"]), dtype, shared=rng.choice(["same", "q8_0"]),
                      skew=rng.random() < 0.7, **shape)
    tokens = _log_int(rng, 1, 64)
    weights = rng.choice(["q4_k", "q4_k", "q8_0", "q5"])
    layout = rng.choice(["planar", "planar", "gguf"]) if weights == "q4_k" else "gguf"
    layers = 1 if weights == "q8_0" or tokens > 16 else (4 if tokens <= 4 else 2)
    return _layer("decode", tokens, weights, layout, dtype, layers=layers, shared="q8_0" if weights == "q5" else "same", **shape)


_TYPES = {"q4_k": (formats.Q4_K, formats.Q4_K), "q8_0": (formats.Q8_0, formats.Q8_0), "q5": (formats.Q5_K, formats.Q5_1)}   # gate / up, down
_LAYOUTS = {"planar": formats.PLANAR, "gguf": formats.GGUF}
_DTYPES = {"f16": torch.float16, "f32": torch.float32}


def _normal(gen, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32).to(dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "head":
        rows, vocab = case["rows"], case["vocabulary"]
        matrix = torch.empty(vocab * (CHANNELS // 32) * 34, dtype=torch.uint8, device="cuda")
        capi.call("tsp_synth_weights", formats.Q8_0, seed, 0, vocab * (CHANNELS // 32), 0.02, matrix.data_ptr(), L.stream_ptr())
        x = _normal(gen, rows, CHANNELS)
        if case["exact"]:
            x = x.half().float()
        return {"case": case, "matrix": matrix, "set": L.matrix_set(matrix, formats.Q8_0, formats.GGUF, vocab, CHANNELS), "x": x,
                "logits": torch.empty(rows, vocab, device="cuda"), "error": torch.zeros(1, dtype=torch.int32, device="cuda")}
    if case["kind"] == "top64":
        rows, vocab, lib = case["rows"], case["vocabulary"], capi.lib()
        return {"case": case, "logits": _normal(gen, rows, vocab),
                "partial": torch.empty(lib.tsp_logit_topk_scratch_bytes(rows, vocab), dtype=torch.uint8, device="cuda"),
                "top": torch.empty(lib.tsp_logit_topk_output_bytes(rows), dtype=torch.uint8, device="cuda")}
    if case["kind"] == "edges":
        t, c, e = case["tokens"], case["channels"], case["experts"]
        return {"case": case, "normalized": _normal(gen, t, BRANCHES, c), "scores": _normal(gen, t, BRANCHES, c), "inject": _normal(gen, t, BRANCHES),
                "streams": _normal(gen, t, BRANCHES, c), "ffn": _normal(gen, t, c), "router": 0.02 * _normal(gen, e, c), "gate_row": 0.02 * _normal(gen, c),
                "rows": torch.empty(t, c, device="cuda"), "scales": torch.empty(t, BRANCHES, device="cuda"), "logits": torch.empty(t, e, device="cuda"),
                "gate": torch.empty(t, device="cuda"), "new_streams": torch.empty(t, BRANCHES, c, device="cuda"),
                "error": torch.zeros(1, dtype=torch.int32, device="cuda")}
    up_type, down_type = _TYPES[case["weights"]]
    dims = (case["channels"], case["hidden"], case["experts"])
    dtype, tokens, n = _DTYPES[case["dtype"]], case["tokens"], case["layers"]
    layers = [L.SynthDeviceLayer(seed * 8 + i, *dims, up_type, _LAYOUTS[case["layout"]], shared_type=formats.Q8_0 if case["shared"] == "q8_0" else None,
                                 down_type=down_type if down_type != up_type else None) for i in range(n)]
    scratch = (L.PrefillScratch if case["kind"] == "prefill" else L.Scratch)(*dims, case["selected"], tokens)
    bias = torch.from_numpy(synth.zipf_bias(seed, case["experts"])).cuda() if case["skew"] else 0.0
    return {"case": case, "layers": layers, "scratch": scratch, "x": [_normal(gen, tokens, dims[0], dtype=dtype) for _ in range(n)],
            "logits": [_normal(gen, tokens, case["experts"]) + bias for _ in range(n)],
            "out": [torch.empty(tokens, dims[0], dtype=dtype, device="cuda") for _ in range(n)]}


def run(state):
    case = state["case"]
    if case["kind"] == "head":
        rows, vocab, logits = case["rows"], case["vocabulary"], state["logits"]
        capi.call("tsp_moe_project", C.byref(state["set"]), state["x"].data_ptr(), CHANNELS * 4, 1, rows, 1, None, None, None, logits.data_ptr(), vocab * 4,
                  int(case["exact"]), state["error"].data_ptr(), L.stream_ptr())
        return logits
    if case["kind"] == "top64":
        rows, vocab, top = case["rows"], case["vocabulary"], state["top"]
        capi.call("tsp_logit_topk", state["logits"].data_ptr(), vocab * 4, rows, vocab, state["partial"].data_ptr(), state["partial"].numel(), top.data_ptr(),
                  top.numel(), L.stream_ptr())
        return top   # rows of four header words, 64 ids and the bits of 64 logits
    if case["kind"] == "edges":
        t, c, e, s, stream = case["tokens"], case["channels"], case["experts"], state, L.stream_ptr()
        error = s["error"].data_ptr()
        capi.call("tsp_residual_read", s["normalized"].data_ptr(), s["scores"].data_ptr(), s["inject"].data_ptr(), BRANCHES, c, t, s["rows"].data_ptr(),
                  s["scales"].data_ptr(), error, stream)
        capi.call("tsp_router_project", s["router"].data_ptr(), e, c, s["gate_row"].data_ptr(), s["rows"].data_ptr(), c * 4, t, s["logits"].data_ptr(), e * 4,
                  s["gate"].data_ptr(), error, stream)
        capi.call("tsp_residual_write", s["streams"].data_ptr(), s["ffn"].data_ptr(), s["scales"].data_ptr(), BRANCHES, c, t, s["new_streams"].data_ptr(),
                  error, stream)
        return [s["rows"], s["scales"], s["logits"], s["gate"], s["new_streams"]]
    step = L.moe_layer_prefill if case["kind"] == "prefill" else L.moe_layer_decode
    for weights, x, logits, out in zip(state["layers"], state["x"], state["logits"], state["out"]):
        step(weights, state["scratch"], x, logits, out)
    return state["out"]


def _experts_hit(case):
    """Distinct routed experts of one batch: a simulated batch of the case's router distribution."""
    rng = np.random.default_rng(1)
    logits = rng.standard_normal((case["tokens"], case["experts"]), dtype=np.float32)
    if case["skew"]:
        logits += synth.zipf_bias(1, case["experts"])
    return len(np.unique(np.argpartition(-logits, case["selected"] - 1, axis=1)[:, :case["selected"]]))


def work(case):
    if case["kind"] == "head":
        m, v = case["rows"], case["vocabulary"]
        return {"bytes": v * (CHANNELS // 32) * 34 + m * CHANNELS * 4 + m * v * 4, "flops": 2 * m * v * CHANNELS}
    if case["kind"] == "top64":
        return {"bytes": case["rows"] * (case["vocabulary"] * 4 + 528), "flops": 0}
    if case["kind"] == "edges":
        t, c, e = case["tokens"], case["channels"], case["experts"]
        wide, narrow = 4 * t * BRANCHES * c, 4 * t * c
        return {"bytes": 4 * wide + 2 * narrow + 4 * (e + 1) * c + 4 * t * (e + 1 + 2 * BRANCHES), "flops": 2 * t * (e + 1) * c + 8 * t * BRANCHES * c}
    t, c, h, k = case["tokens"], case["channels"], case["hidden"], case["selected"]
    up_type, down_type = _TYPES[case["weights"]]
    size = lambda type_: formats.gguf_bytes(type_, h, c)   # noqa: E731
    routed = 2 * size(up_type) + size(down_type)
    shared = 3 * size(formats.Q8_0) if case["shared"] == "q8_0" else routed
    row = 2 if case["dtype"] == "f16" else 4
    once = _experts_hit(case) * routed + shared + 2 * t * c * row + 4 * t * case["experts"] + 4 * c
    return {"bytes": case["layers"] * once, "flops": case["layers"] * t * (k + 1) * 6 * h * c}


def tolerance(case):
    # About four times the distance from the same path in 64 bits over exactly decoded weights, the largest over the listed and a
    # dozen drawn cases: decode 3.4e-6 / 1.8e-5 (relative / largest) with FP32 rows, 2.2e-4 / 4.9e-4 with binary16 rows (their
    # rounding), prefill 6.7e-4 / 5e-3 (binary16 operands), head 2.8e-7 / 1.1e-6 and edges 9e-7 / 5.6e-6 (FP32 sums of 2048 terms).
    if case["kind"] == "top64":
        return "exact"
    if case["kind"] == "head":
        return {"rel": 1.5e-6, "max": 8e-6}
    if case["kind"] == "edges":
        return {"rel": 4e-6, "max": 2.5e-5}
    if case["kind"] == "prefill":
        return {"rel": 2.7e-3, "max": 2e-2}
    return {"rel": 9e-4, "max": 2e-3} if case["dtype"] == "f16" else {"rel": 1.4e-5, "max": 7e-5}
