"""What a program does with this framework all day, as cases that can be timed and compared.

The framework is the quantized-weight matmul of GGUF models (Q8_0, Q4_K, Q6_K). Its user loads or quantizes weights, then
multiplies: one row at a time while it generates text, a few rows at a time for several sequences or speculative tokens, and
hundreds to thousands of rows for a prompt. The cases take that work through the public calls: `QTensor` / `QMatMul`, `ops.*`
for grouped projections, and the launcher pairs that a host of the reference's own call sequence uses.

Weights are real quantizations of N(0, 0.02) values, activations are N(0, 1), both made from the seed on the GPU.
"""
from __future__ import annotations

import torch

import inference_rs_b200 as pkg
from inference_rs_b200 import ops, workloads
from inference_rs_b200.workloads import ModelShape

TYPES = {"q8_0": pkg.GgmlDType.Q8_0, "q4_k": pkg.GgmlDType.Q4K, "q6_k": pkg.GgmlDType.Q6K}
ELEMS = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}

# the largest listed prompt: nothing drawn multiplies more than this
MAX_ROWS_N_K = 8192 * 28672 * 4096
MAX_TOKEN_BYTES = workloads.LLAMA3_8B.weight_bytes_per_token()


def _model(case) -> ModelShape:
    return ModelShape("case", case["layers"], case["hidden"], case["hidden"] // 128, case["kv"] // 128, 128, case["ffn"], case["vocab"])


def _matmul(name, wtype, k, n, rows, dtype):
    return {"name": name, "kind": "matmul", "wtype": wtype, "k": k, "n": n, "rows": rows, "dtype": dtype}


def listed():
    m = workloads.LLAMA3_8B
    shape = {"hidden": m.hidden, "kv": m.kv_heads * m.head_dim, "ffn": m.ffn, "vocab": m.vocab}
    return [
        # Generating one token in a serving loop: all matmuls of the 8B model's step, batch 1, captured once in a CUDA graph and
        # replayed for every token (what bench.py's headline runs).
        {"name": "token_graph", "kind": "token", "graph": True, "layers": m.layers, **shape, "dtype": "bf16"},
        # The same call by call, as a program without graphs makes it: two layers and the output head.
        {"name": "token_calls", "kind": "token", "graph": False, "layers": 2, **shape, "dtype": "bf16"},
        # The smallest call: one row through one small projection (attn_k); latency is all there is.
        _matmul("row_1_small", "q4_k", 4096, 1024, 1, "bf16"),
        # Four sequences decoded together (or four speculative tokens) through the widest layer, gate + up.
        _matmul("rows_4_wide", "q4_k", 4096, 28672, 4, "bf16"),
        # Sixteen sequences through ffn_down: the deep one, in the other K-quant.
        _matmul("rows_16_deep", "q6_k", 14336, 4096, 16, "bf16"),
        # A short prompt of a ragged length in the Q8_0 type, f16 activations, fused q/k/v shape.
        _matmul("prompt_333", "q8_0", 4096, 6144, 333, "f16"),
        # A prompt chunk as schedulers cut them, through ffn_down.
        _matmul("prompt_512_deep", "q6_k", 14336, 4096, 512, "bf16"),
        # A long prompt through gate + up: the largest product.
        _matmul("prompt_8192_wide", "q4_k", 4096, 28672, 8192, "bf16"),
        # The MLP of one decoded token in the reference host's own sequence: quantize the row, fused gate/up with SiLU,
        # quantize, ffn_down.
        {"name": "host_mlp", "kind": "host_mlp", "gate_type": "q4_k", "down_type": "q6_k", "k": 4096, "ffn": 14336, "rows": 1, "dtype": "bf16"},
        # The reference host's prompt sequence: quantize the activations to its prefill blocks, then its matmul launcher.
        {"name": "host_prompt", "kind": "host_prompt", "wtype": "q4_k", "k": 4096, "n": 14336, "rows": 1024, "dtype": "bf16"},
        # Quantizing a weight matrix while a model is loaded (in-situ quantization), ffn_up's shape.
        {"name": "quantize", "kind": "quantize", "wtype": "q4_k", "k": 4096, "n": 14336},
        # The embedding rows of a prompt out of a packed table.
        {"name": "embedding", "kind": "rows", "wtype": "q6_k", "k": 4096, "n": 128256, "ids": 2048, "dtype": "bf16"},
    ]


# ---- the ranges the listed cases stand for -------------------------------------------------------------------------------

def _log_int(rng, lo, hi, step=1):
    return max(lo, int(round(lo * (hi / lo) ** rng.random() / step)) * step)


def _draw_k(rng, wtype, hi):
    if wtype == "q8_0" and rng.random() < 0.25:
        return _log_int(rng, 512, hi, 32)  # whole blocks of 32 are all that Q8_0 asks for
    return _log_int(rng, 512, hi, 256)


def _draw_n(rng, hi):
    return _log_int(rng, 256, hi, rng.choice([1, 8, 64, 256]))


def draw(rng):
    kind = rng.choice(["token", "token", "few", "few", "few", "few", "prompt", "prompt", "prompt", "host_mlp", "host_prompt", "quantize",
                       "rows"])
    wtype, dtype = rng.choice(["q4_k", "q4_k", "q6_k", "q8_0"]), rng.choice(["bf16", "bf16", "bf16", "f16", "f32"])
    if kind == "token":
        while True:
            hidden = _log_int(rng, 1024, 8192, 256)
            case = {"kind": "token", "graph": rng.random() < 0.5, "layers": rng.randint(1, 8), "hidden": hidden,
                    "kv": min(hidden, 128 * rng.choice([4, 8, 8, 16])), "ffn": _log_int(rng, 2 * hidden, 4 * hidden, 256),
                    "vocab": _log_int(rng, 16000, 152064, rng.choice([1, 64])), "dtype": rng.choice(["bf16", "bf16", "f16", "f32"])}
            if _model(case).weight_bytes_per_token() <= MAX_TOKEN_BYTES:
                return case
    if kind == "few":
        return {"kind": "matmul", "wtype": wtype, "k": _draw_k(rng, wtype, 28672), "n": _draw_n(rng, 65536), "rows": _log_int(rng, 1, 16),
                "dtype": dtype}
    if kind == "prompt":
        while True:
            case = {"kind": "matmul", "wtype": wtype, "k": _draw_k(rng, wtype, 16384), "n": _draw_n(rng, 32768), "rows": _log_int(rng, 17, 8192),
                    "dtype": dtype}
            if case["k"] % 64 != 0:
                case["k"] = (case["k"] + 63) // 64 * 64  # the prompt path's step
            if case["rows"] * case["n"] * case["k"] <= MAX_ROWS_N_K:
                return case
    if kind == "host_mlp":
        k = _log_int(rng, 1024, 8192, 256)
        return {"kind": "host_mlp", "gate_type": wtype, "down_type": rng.choice(["q4_k", "q6_k"]), "k": k, "ffn": _log_int(rng, 2 * k, 4 * k, 256),
                "rows": rng.choice([1, 1, 2, 4, 8]), "dtype": dtype}
    if kind == "host_prompt":
        return {"kind": "host_prompt", "wtype": wtype, "k": _log_int(rng, 1024, 14336, 256), "n": _draw_n(rng, 28672),
                "rows": _log_int(rng, 17, 4096), "dtype": dtype}
    if kind == "quantize":
        return {"kind": "quantize", "wtype": wtype, "k": _log_int(rng, 512, 14336, 256), "n": _draw_n(rng, 16384)}
    ids = _log_int(rng, 1, 8192)
    case = {"kind": "rows", "wtype": wtype, "k": _log_int(rng, 1024, 8192, 256), "n": _log_int(rng, 16000, 152064), "ids": ids, "dtype": dtype}
    if rng.random() < 0.4:  # the whole matrix instead of chosen rows
        case["n"], case["ids"] = _draw_n(rng, 28672), 0
    return case


# ---- inputs --------------------------------------------------------------------------------------------------------------

def _weights(wtype, n, k, gen) -> pkg.QTensor:
    w = torch.randn(n, k, device="cuda", generator=gen)
    return pkg.QTensor.quantize(w.mul_(0.02), TYPES[wtype])


def _rolled(q: pkg.QTensor, by: int) -> pkg.QTensor:
    """The same rows in another order, in memory of their own: another layer's matrix without quantizing one more."""
    n, k = q.shape
    data = q.data.clone()
    body = n * q.dtype.row_bytes(k)
    data[:body].view(n, -1).copy_(q.data[:body].view(n, -1).roll(by, 0))
    return pkg.QTensor(data, q.dtype, q.shape)


def _acts(rows, k, dtype, gen) -> torch.Tensor:
    return torch.randn(rows, k, device="cuda", generator=gen).to(ELEMS[dtype])


GROUPS = (("attn_q", "attn_k", "attn_v"), ("attn_output",), ("ffn_gate", "ffn_up"), ("ffn_down",))
INPUTS = ("attn", "mix", "mlp", "down")  # of each group: attn_norm, the attention output, ffn_norm, SiLU(gate) * up


def _grouped(layer, acts):
    """Which matrices go out in one launch: each group that the library takes as a group, the others one by one."""
    plan = []
    for names, i in zip(GROUPS, INPUTS):
        ws = [layer[name] for name in names]
        try:
            if len(ws) > 1:
                ops.gemv_group([w.dtype for w in ws], [w.data for w in ws], acts[i], [w.shape[0] for w in ws])
            plan.append((names, i))
        except pkg.KernelLibraryError as e:
            if e.status != -1:  # not "launch the matrices one by one"
                raise
            plan += [((name,), i) for name in names]
    return plan


def _prepare_token(case, gen):
    model, dtype = _model(case), case["dtype"]
    tag = {v: t for t, v in TYPES.items()}
    projs = model.layer_projections()
    first = {p.name: _weights(tag[p.dtype], p.n, p.k, gen) for p in projs}
    layers = [first] + [{p.name: _rolled(first[p.name], 37 * li) for p in projs} for li in range(1, model.layers)]
    out = model.output_projection()
    head = _weights(tag[out.dtype], out.n, out.k, gen)
    acts = [{"attn": _acts(1, model.hidden, dtype, gen), "mix": _acts(1, model.hidden, dtype, gen), "mlp": _acts(1, model.hidden, dtype, gen),
             "down": _acts(1, model.ffn, dtype, gen)} for _ in range(model.layers)]
    x_head = _acts(1, model.hidden, dtype, gen)
    plan = _grouped(first, acts[0])
    if not case["graph"]:
        calls = [([w[name] for name in names], pkg.QMatMul(w[names[0]]), x[i]) for w, x in zip(layers, acts) for names, i in plan]
        return {"kind": "token", "graph": None, "calls": calls + [([head], pkg.QMatMul(head), x_head)]}
    # a decoder sets its launch mode and the order of its matrices once, runs a step, and captures it
    outs = {p.name: torch.empty(model.layers, p.n, dtype=ELEMS[dtype], device="cuda") for p in projs}
    logits = torch.empty(1, out.n, dtype=ELEMS[dtype], device="cuda")
    launches = [([w[name] for name in names], x[i], [outs[name][li:li + 1] for name in names])
                for li, (w, x) in enumerate(zip(layers, acts)) for names, i in plan]
    launches.append(([head], x_head, [logits]))

    def step():
        for ws, x, dst in launches:
            if len(ws) > 1:
                ops.gemv_group([w.dtype for w in ws], [w.data for w in ws], x, [w.shape[0] for w in ws], outs=dst)
            else:
                ops.gemv(ws[0].dtype, ws[0].data, x, ws[0].shape[0], out=dst[0])

    torch.cuda.synchronize()  # the weights are there before the first early-started launch reads them
    ops.set_option("pdl", 1)
    for (ws, _, _), (nxt, _, _) in zip(launches, launches[1:] + launches[:1]):
        ops.set_weight_successor(ws[-1].data, nxt[0].data, nxt[0].dtype, nxt[0].shape[1], nxt[0].shape[0])
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        step()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            step()
    torch.cuda.synchronize()
    ops.clear_weight_successors()
    ops.set_option("pdl", 0)
    return {"kind": "token", "graph": graph, "launches": launches, "outs": outs, "logits": logits}


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "token":
        return _prepare_token(case, gen)
    if kind == "matmul":
        w = pkg.QMatMul(_weights(case["wtype"], case["n"], case["k"], gen))
        return {"kind": kind, "w": w, "x": _acts(case["rows"], case["k"], case["dtype"], gen)}
    if kind == "host_mlp":
        gate, up = (_weights(case["gate_type"], case["ffn"], case["k"], gen) for _ in range(2))
        down = _weights(case["down_type"], case["k"], case["ffn"], gen)
        return {"kind": kind, "gate": gate, "up": up, "down": down, "x": _acts(case["rows"], case["k"], case["dtype"], gen)}
    if kind == "host_prompt":
        return {"kind": kind, "w": _weights(case["wtype"], case["n"], case["k"], gen), "x": _acts(case["rows"], case["k"], case["dtype"], gen)}
    if kind == "quantize":
        return {"kind": kind, "dtype": TYPES[case["wtype"]], "src": torch.randn(case["n"], case["k"], device="cuda", generator=gen).mul_(0.02)}
    w = _weights(case["wtype"], case["n"], case["k"], gen)
    ids = torch.randint(0, case["n"], (case["ids"],), device="cuda", generator=gen, dtype=torch.int32) if case["ids"] else None
    return {"kind": kind, "w": w, "ids": ids, "dtype": ELEMS[case["dtype"]]}


# ---- one pass ------------------------------------------------------------------------------------------------------------

def _run_token_calls(s):
    outs = []
    for ws, mat, x in s["calls"]:
        if len(ws) > 1:
            outs += ops.gemv_group([w.dtype for w in ws], [w.data for w in ws], x, [w.shape[0] for w in ws])
        else:
            outs.append(mat.forward(x))
    return outs


def run(s):
    kind = s["kind"]
    if kind == "token":
        if s["graph"] is None:
            return _run_token_calls(s)
        s["graph"].replay()
        return {"logits": s["logits"], **s["outs"]}
    if kind == "matmul":
        return s["w"].forward(s["x"])
    if kind == "host_mlp":
        x, gate, up, down = s["x"], s["gate"], s["up"], s["down"]
        ffn, k = gate.shape
        h = ops.mmvq_fused_glu(gate.dtype, gate.data, up.data, ops.quantize_q8_1(x), ffn, k, x.shape[0], x.dtype)
        return ops.mmvq_plain(down.dtype, down.data, ops.quantize_q8_1(h), k, ffn, x.shape[0], x.dtype)
    if kind == "host_prompt":
        w, x = s["w"], s["x"]
        n, k = w.shape
        return ops.mmq(w.dtype, w.data, ops.quantize_mmq_q8_1(x, ops.MMQ_LAYOUT[w.dtype]), x.shape[0], n, k, x.dtype)
    if kind == "quantize":
        return pkg.QTensor.quantize(s["src"], s["dtype"]).packed_bytes()
    if s["ids"] is None:
        return s["w"].dequantize(s["dtype"])
    return s["w"].embedding(s["ids"], s["dtype"])


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "token":
        es, model = ELEMS[case["dtype"]].itemsize, _model(case)
        projs = model.layer_projections()
        acts = model.layers * (3 * model.hidden + model.ffn) + model.hidden
        outs = model.layers * sum(p.n for p in projs) + model.vocab
        values = model.layers * sum(p.n * p.k for p in projs) + model.vocab * model.hidden
        return {"bytes": model.weight_bytes_per_token() + es * (acts + outs), "flops": 2 * values}
    if kind == "host_mlp":
        es, k, ffn, rows = ELEMS[case["dtype"]].itemsize, case["k"], case["ffn"], case["rows"]
        packed = 2 * ffn * TYPES[case["gate_type"]].row_bytes(k) + k * TYPES[case["down_type"]].row_bytes(ffn)
        return {"bytes": packed + 2 * es * rows * k, "flops": 2 * rows * 3 * k * ffn}
    t, n, k = TYPES[case["wtype"]], case["n"], case["k"]
    if kind == "quantize":
        return {"bytes": 4 * n * k + n * t.row_bytes(k), "flops": 0}
    es = ELEMS[case["dtype"]].itemsize
    if kind == "rows":
        count = case["ids"] or n
        return {"bytes": count * (t.row_bytes(k) + es * k) + 4 * case["ids"], "flops": 0}
    return {"bytes": n * t.row_bytes(k) + es * case["rows"] * (k + n), "flops": 2 * case["rows"] * n * k}


def tolerance(case):
    kind = case["kind"]
    if kind in ("quantize", "rows"):
        return "exact"  # packed bytes, and values that have one correct rounding
    if case["dtype"] == "f32" and kind == "host_mlp":
        return {"rel": 1e-3}  # the middle of the MLP is quantized to 8 bits again: a last-bit difference can move a whole step
    if case["dtype"] == "f32" and (kind == "token" or (kind == "matmul" and case["rows"] <= 8)):
        return {"rel": 1e-5}  # exact integer dot products, 32-bit sums
    if case["dtype"] == "f32" and kind == "matmul" and case["rows"] <= 16 and pkg.qmatmul.tensor_core_rows_supported(TYPES[case["wtype"]], case["k"]):
        return {"rel": 1e-5}  # the same up to 16 rows where packed rows are whole 16-byte pieces; 16-bit operands elsewhere
    if case["dtype"] == "f16" and kind in ("token", "matmul"):
        return {"rel": 2e-3}
    return {"rel": 1e-2}  # bf16 results, or bf16 operands under f32 results
