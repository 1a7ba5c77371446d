"""The work whose speed this repository answers for: passes through the quantized linears of a decoder.

A case is one decoder's linear stack (hidden size, projections, layers, quantization mix, output head),
a number of activation rows and the way a program drives it:

  "graph"   decoding as a server does it: the pass is captured once in a CUDA graph and replayed per token
  "eager"   calls issued one by one, outputs allocated by the calls: prefill, where a call is long
  "linears" one LinearX.forward per projection with its bias, nothing batched or captured: the first
            program anybody writes, bound by what a call costs
  "fused"   the fused neighbours in a captured decode pass: embedding lookup, RMSNorm in front of the
            projections, SwiGLU behind gate|up, top-k behind the head
  "host"    a decoder that keeps its activations in page-locked host memory (bound host calls)

Modes are the defaults: up to 16 rows the integer scheme, above it the tensor-core scheme. Every layer
has its own weights, inputs and outputs. Weights are N(0, 0.02) quantized by the library's own quantizer,
activations N(0, 1): what the linears of a normalised transformer see.
"""
import math

import torch

import tur_b200 as tq
from tur_b200.workloads import BLOCK, Q4_K, Q5_K, Q6_K, Q8_0, WORKLOADS, quantized_blocks

TOPK = 40        # candidates a sampler keeps
EPS = 1e-6
MAIN = {"q8_0": (Q8_0, Q8_0), "q4_k_m": (Q4_K, Q6_K), "q5_k_m": (Q5_K, Q6_K)}  # projections | attn_v, ffn_down, head


def _case(name, shape, mix, layers, rows, drive, x="f32", head=False):
    w = WORKLOADS[shape]
    by = {p.name: p for p in w.per_layer}
    return {"name": name, "hidden": w.hidden, "q_out": by["attn_q"].n, "kv_out": by["attn_k"].n, "inter": by["ffn_gate"].n,
            "vocab": 151936 if head else 0, "mix": mix, "layers": layers, "rows": rows, "drive": drive, "x": x}


def listed():
    return [
        # one token of a 0.6B model: 112 launches of 1-7 MB, latency and launch gaps are everything
        _case("decode_0.6b_q8_m1", "cfg1", "q8_0", 28, 1, "graph"),
        # the same model driven call by call, as a first program does
        _case("linears_0.6b_q8_m1", "cfg1", "q8_0", 4, 1, "linears"),
        # one token of an 8B model, head included: the single-user decode everything is quoted on
        _case("decode_8b_q4km_m1", "cfg2", "q4_k_m", 36, 1, "graph", head=True),
        # the same token for a program that keeps activations on the host
        _case("host_8b_q4km_m1", "cfg2", "q4_k_m", 12, 1, "host"),
        # a few users at once through the fused entries, logits to candidates
        _case("fused_8b_q4km_m8", "cfg2", "q4_k_m", 8, 8, "fused", head=True),
        # a full small batch: the last row count of the integer scheme
        _case("decode_8b_q4km_m16", "cfg2", "q4_k_m", 12, 16, "graph"),
        # continuous batching on a 3B model and on a 32B model
        _case("decode_3b_q5km_m32", "cfg4-q5", "q5_k_m", 40, 32, "graph"),
        _case("decode_32b_q4km_m64", "cfg5", "q4_k_m", 8, 64, "graph"),
        # prefill: a short prompt, one that is no multiple of any tile, a long one, a chunk of a big model
        _case("prefill_8b_q4km_m512", "cfg2", "q4_k_m", 4, 512, "eager", x="bf16"),
        _case("prefill_3b_q8_m1000", "cfg4-q8", "q8_0", 4, 1000, "eager", x="bf16"),
        _case("prefill_8b_q5km_m2048", "cfg3-q5", "q5_k_m", 2, 2048, "eager", x="bf16"),
        _case("prefill_32b_q4km_m4096", "cfg5", "q4_k_m", 1, 4096, "eager", x="bf16"),
    ]


def draw(rng):
    """Any of the drives at sizes spread over the listed range, odd ones among them: projection widths,
    vocabularies and row counts that divide by nothing in particular."""
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    drive = rng.choice(["graph", "graph", "graph", "eager", "eager", "linears", "fused", "host"])
    mix = rng.choice(["q8_0", "q4_k_m", "q5_k_m"])
    block = 64 if mix == "q8_0" else 256      # in-features are whole blocks
    hidden = max(block, round(log(768, 5120) / block) * block)
    inter = max(block, round(hidden * rng.uniform(2.5, 5.0) / block) * block)
    q_out = max(block, round(hidden * rng.choice([1.0, 1.0, 1.6, 2.0]) / block) * block)
    kv_out = max(8, round(hidden * rng.choice([1.0, 0.5, 0.25, 0.125]) / 8) * 8)
    rows = {"graph": lambda: round(log(1, 128)), "eager": lambda: round(log(65, 8192)), "linears": lambda: round(log(1, 64)),
            "fused": lambda: round(log(1, 32)), "host": lambda: round(log(1, 16))}[drive]()
    head = drive == "fused" or (drive == "graph" and rng.random() < 0.3)
    c = {"hidden": hidden, "q_out": q_out, "kv_out": kv_out, "inter": inter, "vocab": round(log(20000, 152000)) if head else 0,
         "mix": mix, "layers": 1, "rows": rows, "drive": drive, "x": "bf16" if drive == "eager" or rng.random() < 0.25 else "f32"}
    if drive == "host":
        c["x"] = "f32"
    weight_bytes = sum(_bytes(n, k, dt) for _, n, k, dt, _ in _linears(c))
    flops = sum(2 * rows * n * k for _, n, k, dt, _ in _linears(c))
    most = min(1.5e9 / weight_bytes, 1.5e12 / flops, 4 if drive in ("eager", "linears") else 8 if drive == "fused" else 24)
    c["layers"] = max(1, int(most))
    return c


# ---- the stack of a case

def _linears(c):
    """(name, out-features, in-features, type, the input that feeds it) of one layer."""
    main, alt = MAIN[c["mix"]]
    h, q, kv, f = c["hidden"], c["q_out"], c["kv_out"], c["inter"]
    return [("attn_q", q, h, main, "hidden"), ("attn_k", kv, h, main, "hidden"), ("attn_v", kv, h, alt, "hidden"),
            ("attn_output", h, q, main, "attn"), ("ffn_gate", f, h, main, "mlp"), ("ffn_up", f, h, main, "mlp"),
            ("ffn_down", h, f, alt, "inter")]


def _bytes(n, k, dt):
    be, bb = BLOCK[dt]
    return n * (k // be) * bb


def _weight(n, k, dt, seed):
    return tq.QMatMul.from_arc(tq.QTensor.new(quantized_blocks(dt, n, k, seed, torch.device("cuda", 0)), tq.GgmlDType(dt), (n, k)))


GROUPS = (("attn_q", "attn_k", "attn_v"), ("attn_output",), ("ffn_gate", "ffn_up"), ("ffn_down",))  # linears that share an input


def prepare(case, seed):
    dev = torch.device("cuda", 0)
    rows, layers, drive = case["rows"], case["layers"], case["drive"]
    lin = _linears(case)
    gen = torch.Generator(device=dev).manual_seed(seed * 7919 + 1)
    xdt = torch.bfloat16 if case["x"] == "bf16" else torch.float32

    def randn(*shape):
        return torch.randn(shape, device=dev, generator=gen)

    s = {"case": case, "layers": []}
    dims = {"hidden": case["hidden"], "attn": case["q_out"], "mlp": case["hidden"], "inter": case["inter"]}
    for i in range(layers):
        lay = {"w": {name: _weight(n, k, dt, seed * 1000003 + 16 * i + j) for j, (name, n, k, dt, _) in enumerate(lin)},
               "x": {src: randn(rows, d).to(xdt) for src, d in dims.items()}}
        if drive == "linears":
            lay["linear"] = {name: tq.LinearX(lay["w"][name], randn(n) * 0.1) for name, n, *_ in lin}
        if drive == "fused":
            lay["norm"] = {"hidden": 1 + 0.1 * randn(case["hidden"])}
        s["layers"].append(lay)
    if case["vocab"]:
        s["head"] = _weight(case["vocab"], case["hidden"], MAIN[case["mix"]][1], seed * 1000003 + 999)
        s["x_head"] = randn(rows, case["hidden"]).to(xdt)
    if drive == "fused":
        s["table"] = _weight(case["vocab"], case["hidden"], MAIN[case["mix"]][0], seed * 1000003 + 998).qtensor
        s["ids"] = torch.randint(0, case["vocab"], (rows,), device=dev, dtype=torch.int32, generator=gen)
    if drive == "host":
        s["y"] = {name: torch.zeros((layers, rows, n), dtype=torch.float32).pin_memory() for name, n, *_ in lin}
        s["calls"] = []
        for i, lay in enumerate(s["layers"]):
            for g in GROUPS:
                src = next(l[4] for l in lin if l[0] == g[0])
                x = lay["x"][src].float().cpu().pin_memory()
                s["calls"].append(tq.HostCall([lay["w"][name] for name in g], x, [s["y"][name][i] for name in g]))
    if drive in ("graph", "fused"):
        if drive == "graph":
            s["y"] = {name: torch.zeros((layers, rows, n), dtype=torch.float32, device=dev) for name, n, *_ in lin}
            if case["vocab"]:
                s["y"]["head"] = torch.zeros((rows, case["vocab"]), dtype=torch.float32, device=dev)
        step = _decode_step if drive == "graph" else _fused_step
        tq.context(0).reserve(rows, max(dims.values()), max([case["vocab"]] + [l[1] for l in lin]))
        stream = torch.cuda.Stream(dev)
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            step(s)
        torch.cuda.current_stream().wait_stream(stream)
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"], stream=stream):
            s["out"] = step(s)
    return s


def _decode_step(s):
    for i, lay in enumerate(s["layers"]):
        w, x = lay["w"], lay["x"]
        tq.QMatMul.forward_multi([w[n] for n in GROUPS[0]], x["hidden"], outs=[s["y"][n][i] for n in GROUPS[0]])
        w["attn_output"].forward(x["attn"], out=s["y"]["attn_output"][i])
        tq.QMatMul.forward_multi([w[n] for n in GROUPS[2]], x["mlp"], outs=[s["y"][n][i] for n in GROUPS[2]])
        w["ffn_down"].forward(x["inter"], out=s["y"]["ffn_down"][i])
    if "head" in s:
        s["head"].forward(s["x_head"], out=s["y"]["head"])
    return s["y"]


def _fused_step(s):
    out = [s["table"].embedding(s["ids"])]
    for lay in s["layers"]:
        w, x = lay["w"], lay["x"]
        out += tq.QMatMul.rmsnorm_forward_multi([w[n] for n in GROUPS[0]], x["hidden"], lay["norm"]["hidden"], EPS)
        out.append(w["attn_output"].forward(x["attn"]))
        h = tq.QMatMul.swiglu(w["ffn_gate"], w["ffn_up"], x["mlp"])
        out += [h, w["ffn_down"].forward(x["inter"])]
    logits = torch.empty((s["case"]["rows"], s["case"]["vocab"]), dtype=torch.float32, device=s["x_head"].device)
    out += s["head"].lm_head_topk(s["x_head"], k=TOPK, logits_out=logits)
    return out + [logits]


def run(state):
    drive = state["case"]["drive"]
    if drive in ("graph", "fused"):
        state["graph"].replay()
        return state["out"]
    if drive == "host":
        for call in state["calls"]:
            call.run()
        return state["y"]
    out = []
    for lay in state["layers"]:
        x = lay["x"]
        if drive == "linears":
            lin = lay["linear"]
            out += [lin["attn_q"].forward(x["hidden"]), lin["attn_k"].forward(x["hidden"]), lin["attn_v"].forward(x["hidden"]),
                    lin["attn_output"].forward(x["attn"]), lin["ffn_gate"].forward(x["mlp"]), lin["ffn_up"].forward(x["mlp"]),
                    lin["ffn_down"].forward(x["inter"])]
        else:
            w = lay["w"]
            out += tq.QMatMul.forward_multi([w[n] for n in GROUPS[0]], x["hidden"])
            out.append(w["attn_output"].forward(x["attn"]))
            out += tq.QMatMul.forward_multi([w[n] for n in GROUPS[2]], x["mlp"])
            out.append(w["ffn_down"].forward(x["inter"]))
    return out


def work(case):
    """Weights once, every distinct input once, every output once; two operations per weight and row."""
    rows, xb = case["rows"], 2 if case["x"] == "bf16" else 4
    lin = _linears(case)
    outs = sum(n for name, n, *_ in lin if not (case["drive"] == "fused" and name == "ffn_up"))
    per = sum(_bytes(n, k, dt) for _, n, k, dt, _ in lin) + rows * (2 * case["hidden"] + case["q_out"] + case["inter"]) * xb + rows * outs * 4
    flops = sum(2 * rows * n * k for _, n, k, _, _ in lin)
    total, fl = case["layers"] * per, case["layers"] * flops
    if case["vocab"]:
        alt = MAIN[case["mix"]][1]
        total += _bytes(case["vocab"], case["hidden"], alt) + rows * case["hidden"] * xb + rows * case["vocab"] * 4
        fl += 2 * rows * case["vocab"] * case["hidden"]
    if case["drive"] == "fused":
        total += _bytes(rows, case["hidden"], MAIN[case["mix"]][0]) + rows * case["hidden"] * 4
    return {"bytes": total, "flops": fl}


def tolerance(case):
    """Integer scheme: the integers are exact, only f32 sums over the blocks are ordered freely (measured 1.6e-7).
    Behind an RMSNorm an activation can round to the neighbouring int8, and equal-ish logits can change places.
    Tensor-core scheme: f16 operands, measured 3e-4 to 5e-4 from the product in 64 bits."""
    if case["rows"] > 16:
        t = {"rel": 2e-3, "max": 1e-2}
    elif case["drive"] == "fused":
        t = {"rel": 2e-4, "max": 1e-2}
    else:
        t = {"rel": 1e-6, "max": 2e-5}
    if case["drive"] == "fused":
        t["differ"] = 0.01
    return t
