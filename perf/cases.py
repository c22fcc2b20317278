"""The workloads this package is timed on: its public entry points over the sizes they serve.

Shapes come from the benchmark (decode 16 x 7168 x 2048, prefill 4096 x 7168 x 18432 and 8192 x 28672 x 8192, the
row-parallel shard 4096 x 8192 x 3584, the grouped 4 x 2048 rows), the tests and their neighbourhood.  Activations are
standard normal with 1 % of the channels scaled by 20, weights 0.02 x normal.

Every case names its entry point in "op":
  decode_step   a CUDA graph of fp8_linear pairs, the second fed by the first: how the layers of a decoding step are served
  gemm          gemm_fp8_fp8_bf16_nt on quantized operands (the activations arrive quantized by an earlier kernel)
  linear        fp8_linear: bf16 activations in, quantizer + GEMM
  gemm_f32      gemm_fp8_fp8_f32_nt: the partial sums of a row-parallel layer
  gemm_e4m3     gemm_fp8_fp8_e4m3_nt: the GEMM that hands quantized activations to the next layer
  quantize      per_token_cast_to_fp8
  contiguous    m_grouped_gemm_fp8_fp8_bf16_nt_contiguous: mixture-of-experts prefill
  masked        m_grouped_gemm_fp8_fp8_bf16_nt_masked: mixture-of-experts decode
"""
import math
import random

import torch

import yan_b200

F8 = torch.float8_e4m3fn


def listed():
    return [
        # one decoding step of 8 two-matrix layers at 16 sequences, replayed as a graph: launch chains and latency (each
        # layer has an activation of its own: rounding would otherwise grow from layer to layer and hide a wrong result)
        {"name": "decode_step_16", "op": "decode_step", "m": 16, "n": 7168, "k": 2048, "layers": 8},
        # a single sequence through one long-K projection, called eagerly: the smallest call
        {"name": "gemm_1x4096x7168", "op": "gemm", "m": 1, "n": 4096, "k": 7168},
        # the larger decode batch, called eagerly
        {"name": "gemm_64x7168x2048", "op": "gemm", "m": 64, "n": 7168, "k": 2048},
        # a small layer, bf16 in and out
        {"name": "linear_256x1024x1024", "op": "linear", "m": 256, "n": 1024, "k": 1024},
        # a ragged prompt and a width that no tile divides
        {"name": "gemm_1111x5136x3072", "op": "gemm", "m": 1111, "n": 5136, "k": 3072},
        # one rank's share of a row-parallel layer, fp32 partial sums out
        {"name": "f32_4096x8192x3584", "op": "gemm_f32", "m": 4096, "n": 8192, "k": 3584},
        # prefill with long K
        {"name": "gemm_4096x7168x18432", "op": "gemm", "m": 4096, "n": 7168, "k": 18432},
        # the headline prefill layer: quantize the activations, multiply
        {"name": "linear_8192x28672x8192", "op": "linear", "m": 8192, "n": 28672, "k": 8192},
        # the first of two chained layers: codes and scales out
        {"name": "e4m3_8192x7168x2048", "op": "gemm_e4m3", "m": 8192, "n": 7168, "k": 2048},
        # the activation quantizer alone
        {"name": "quantize_8192x8192", "op": "quantize", "m": 8192, "k": 8192},
        # mixture-of-experts prefill: four experts of unequal load, each padded to whole 128-row tiles
        {"name": "contiguous_4x2048", "op": "contiguous", "groups": 4, "rows": 2048, "n": 7168, "k": 2048},
        # mixture-of-experts decode: many experts, a few rows each
        {"name": "masked_16x128", "op": "masked", "groups": 16, "m_max": 128, "rows": 24, "n": 7168, "k": 2048},
    ]


def _log(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng: random.Random):
    """One more case of the same ranges; never more work than the largest listed one."""
    while True:
        op = rng.choice(["decode_step", "gemm", "gemm", "gemm", "linear", "linear", "gemm_f32", "gemm_e4m3", "quantize",
                         "contiguous", "masked"])
        if op == "decode_step":
            case = {"op": op, "m": _log(rng, 1, 64), "n": _log(rng, 1024, 8192, 128), "k": _log(rng, 512, 8192, 128),
                    "layers": rng.randint(2, 8)}
        elif op in ("gemm", "linear"):
            case = {"op": op, "m": _log(rng, 1, 8192), "n": _log(rng, 256, 28672, 16), "k": _log(rng, 256, 18432, 128)}
        elif op == "gemm_f32":
            case = {"op": op, "m": _log(rng, 64, 8192), "n": _log(rng, 512, 8192, 16), "k": _log(rng, 512, 14336, 128)}
        elif op == "gemm_e4m3":
            case = {"op": op, "m": _log(rng, 64, 8192), "n": _log(rng, 512, 14336, 128), "k": _log(rng, 512, 8192, 128)}
        elif op == "quantize":
            case = {"op": op, "m": _log(rng, 1, 16384), "k": _log(rng, 512, 18432, 128)}
        elif op == "contiguous":
            case = {"op": op, "groups": rng.randint(2, 16), "rows": _log(rng, 128, 2048), "n": _log(rng, 512, 8192, 128),
                    "k": _log(rng, 512, 8192, 128)}
        else:
            m_max = rng.choice([64, 128, 256])
            case = {"op": op, "groups": rng.randint(2, 24), "m_max": m_max, "rows": rng.randint(1, m_max),
                    "n": _log(rng, 512, 8192, 128), "k": _log(rng, 512, 8192, 128)}
        w = work(case)
        if w["flops"] <= 3.9e12 and w["bytes"] <= 1.2e9 and case.get("groups", 1) * case.get("n", 1) * case["k"] <= 4.0e8:
            return case


# ---- inputs -------------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(gen, rows, k):
    x = torch.randn(rows, k, generator=gen, device="cuda", dtype=torch.float32)
    x[:, torch.randperm(k, generator=gen, device="cuda")[:max(1, k // 100)]] *= 20.0
    return x.to(torch.bfloat16)


def _weights(gen, n, k):
    """bf16 [n, k] with n rounded up to whole 128-row blocks: the last block of a ragged width is cut after quantizing."""
    n_up = (n + 127) // 128 * 128
    w = torch.empty(n_up, k, dtype=torch.bfloat16, device="cuda")
    for r in range(0, n_up, 4096):
        rows = min(4096, n_up - r)
        w[r:r + rows] = (torch.randn(rows, k, generator=gen, device="cuda", dtype=torch.float32) * 0.02).to(torch.bfloat16)
    return w


def _masked_rows(case, seed):
    rng = random.Random(seed * 7919 + 1)
    return [min(case["m_max"], max(0, int(rng.gauss(case["rows"], case["rows"] / 3)))) for _ in range(case["groups"])]


def _contiguous_rows(case):
    """Valid rows per group, around case["rows"] on average (the same for every seed: they set the output's shape)."""
    rng = random.Random(case["groups"] * 7919 + case["rows"])
    share = [rng.uniform(0.5, 1.5) for _ in range(case["groups"])]
    total = case["rows"] * case["groups"]
    return [max(1, int(total * s / sum(share))) for s in share]


def _inputs(case, seed):
    """The bf16 inputs, from the seed alone."""
    gen, op = _gen(seed), case["op"]
    if op == "quantize":
        return {"x": _activations(gen, case["m"], case["k"])}
    if op == "decode_step":
        x, w = [], []
        for _ in range(case["layers"]):
            x.append(_activations(gen, case["m"], case["k"]))
            w += [_weights(gen, case["n"], case["k"]), _weights(gen, case["k"], case["n"])]
        return {"x": x, "w": w}
    if op == "contiguous":
        rows = _contiguous_rows(case)
        padded = [(r + 127) // 128 * 128 for r in rows]
        return {"x": _activations(gen, sum(padded), case["k"]), "padded": padded,
                "w": [_weights(gen, case["n"], case["k"]) for _ in range(case["groups"])]}
    if op == "masked":
        return {"x": _activations(gen, case["groups"] * case["m_max"], case["k"]), "rows": _masked_rows(case, seed),
                "w": [_weights(gen, case["n"], case["k"]) for _ in range(case["groups"])]}
    return {"x": _activations(gen, case["m"], case["k"]), "w": _weights(gen, case["n"], case["k"])}


def _cast_weights(w, n):
    q, s = yan_b200.per_block_cast_to_fp8(w)
    return (q if q.shape[0] == n else q[:n].contiguous()), s


def _cast_experts(ws):
    pairs = [yan_b200.per_block_cast_to_fp8(w) for w in ws]
    return torch.stack([q.view(torch.uint8) for q, _ in pairs]).view(F8), torch.stack([s for _, s in pairs])


def _empty(*shape, dtype=torch.bfloat16):
    return torch.empty(*shape, dtype=dtype, device="cuda")


def prepare(case, seed):
    op, k = case["op"], case["k"]
    i = _inputs(case, seed)
    st = {"op": op}
    if op == "quantize":
        st["x"] = i["x"]
        st["out"] = (_empty(case["m"], k, dtype=F8), _empty(k // 128, case["m"], dtype=torch.float32).t())
        return st
    if op == "linear":
        st["x"], st["rhs"] = i["x"], _cast_weights(i["w"], case["n"])
        st["out"] = _empty(case["m"], case["n"])
        return st
    if op == "decode_step":
        st["x"] = i["x"]
        widths = [case["n"], case["k"]] * case["layers"]
        st["rhs"] = [_cast_weights(w, n) for w, n in zip(i["w"], widths)]
        st["outs"] = [_empty(case["m"], n) for n in widths]
        need = max(yan_b200.fp8_linear_workspace_bytes(case["m"], kk) for kk in (case["n"], case["k"]))
        st["workspace"] = _empty(need, dtype=torch.uint8)

        def step():
            for j, x in enumerate(st["x"]):
                for l in (2 * j, 2 * j + 1):
                    x = yan_b200.fp8_linear(x, st["rhs"][l], st["outs"][l], workspace=st["workspace"])

        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()  # first calls load kernels, which a capture must not do
        torch.cuda.current_stream().wait_stream(side)
        st["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st["graph"]):
            step()
        return st
    if op == "contiguous":
        st["lhs"] = yan_b200.per_token_cast_to_fp8(i["x"])
        st["rhs"] = _cast_experts(i["w"])
        idx = [g for g, p in enumerate(i["padded"]) for _ in range(p)]
        st["m_indices"] = torch.tensor(idx, dtype=torch.int32, device="cuda")
        st["out"] = _empty(i["x"].shape[0], case["n"]).zero_()
        return st
    if op == "masked":
        g, m_max = case["groups"], case["m_max"]
        q, s = yan_b200.per_token_cast_to_fp8(i["x"])
        # the scales stay as the quantizer laid them out: k-block-major over all rows of all groups
        st["lhs"] = (q.view(g, m_max, k), s.as_strided((g, m_max, k // 128), (m_max, 1, g * m_max)))
        st["rhs"] = _cast_experts(i["w"])
        st["masked_m"] = torch.tensor(i["rows"], dtype=torch.int32, device="cuda")
        st["expected_m"] = case["rows"]
        st["out"] = _empty(g, m_max, case["n"]).zero_()
        return st
    st["lhs"], st["rhs"] = yan_b200.per_token_cast_to_fp8(i["x"]), _cast_weights(i["w"], case["n"])
    m, n = case["m"], case["n"]
    if op == "gemm_e4m3":
        st["out"] = (_empty(m, n, dtype=F8), _empty(n // 128, m, dtype=torch.float32).t())
    else:
        st["out"] = _empty(m, n, dtype=torch.float32 if op == "gemm_f32" else torch.bfloat16)
    return st


def run(st):
    op = st["op"]
    if op == "decode_step":
        st["graph"].replay()
        return st["outs"]
    if op == "gemm":
        yan_b200.gemm_fp8_fp8_bf16_nt(st["lhs"], st["rhs"], st["out"])
    elif op == "linear":
        yan_b200.fp8_linear(st["x"], st["rhs"], st["out"])
    elif op == "gemm_f32":
        yan_b200.gemm_fp8_fp8_f32_nt(st["lhs"], st["rhs"], st["out"])
    elif op == "gemm_e4m3":
        yan_b200.gemm_fp8_fp8_e4m3_nt(st["lhs"], st["rhs"], st["out"])
    elif op == "quantize":
        yan_b200.per_token_cast_to_fp8(st["x"], out=st["out"])
    elif op == "contiguous":
        yan_b200.m_grouped_gemm_fp8_fp8_bf16_nt_contiguous(st["lhs"], st["rhs"], st["out"], st["m_indices"])
    else:
        yan_b200.m_grouped_gemm_fp8_fp8_bf16_nt_masked(st["lhs"], st["rhs"], st["out"], st["masked_m"],
                                                       expected_m=st["expected_m"])
    return st["out"]


# ---- work, tolerance, 64-bit values ---------------------------------------------------------------------------------

def _gemm_bytes(m, n, k, in_bytes, out_bytes):
    """Activations (with their scales where they arrive quantized), weights, block scales, output."""
    scales = 4 * m * (k // 128) if in_bytes == 1 else 0
    return in_bytes * m * k + scales + n * k + 4 * ((n + 127) // 128) * (k // 128) + out_bytes * m * n


def work(case):
    op, k = case["op"], case["k"]
    if op == "quantize":
        return {"bytes": 3 * case["m"] * k + 4 * case["m"] * (k // 128), "flops": 2 * case["m"] * k}
    n = case["n"]
    if op == "decode_step":
        m, layers = case["m"], case["layers"]
        both = _gemm_bytes(m, n, k, 2, 2) + _gemm_bytes(m, k, n, 2, 2)
        return {"bytes": layers * both, "flops": layers * 4 * m * n * k}
    if op in ("contiguous", "masked"):
        rows = case["groups"] * case["rows"]
        one_expert = _gemm_bytes(0, n, k, 1, 2)
        return {"bytes": case["groups"] * one_expert + _gemm_bytes(rows, 0, k, 1, 2) + 2 * rows * n, "flops": 2 * rows * n * k}
    m = case["m"]
    if op == "gemm_e4m3":
        return {"bytes": _gemm_bytes(m, n, k, 1, 1) + 4 * m * (n // 128), "flops": 2 * m * n * k}
    return {"bytes": _gemm_bytes(m, n, k, 2 if op == "linear" else 1, 4 if op == "gemm_f32" else 2), "flops": 2 * m * n * k}


def tolerance(case):
    op = case["op"]
    if op == "quantize":
        return "exact"  # codes and scales are defined operation by operation
    if op == "gemm_f32":
        return {"rel": 1e-6, "max": 1e-5}
    if op == "decode_step":
        return {"rel": 2e-3, "max": 0.05}  # a value of the first product on the other side of a tie reaches all of the second
    if op == "gemm_e4m3":
        return {"rel": 1e-3, "max": 0.15}  # a value that lands on the other side of a tie moves by one e4m3 step
    return {"rel": 2e-4, "max": 0.0157}  # bf16 results whose last bit depends on the order of the sums


def _q_act(x):
    """1 x 128 groups: (e4m3 values as fp32, fp32 scales), each step one fp32 operation."""
    m, k = x.shape
    xf = x.float().view(m, k // 128, 128)
    amax = xf.abs().amax(dim=2).clamp_min(1e-4)
    inv = torch.full_like(amax, 448.0) / amax
    return (xf * inv.unsqueeze(2)).to(F8).float().view(m, k), amax / torch.full_like(amax, 448.0)


def _deq_act(x):
    q, s = _q_act(x)
    m, k = q.shape
    return (q.double().view(m, k // 128, 128) * s.double().unsqueeze(2)).view(m, k)


def _deq_w(w, n):
    """128 x 128 blocks, dequantized in 64 bits."""
    n_up, k = w.shape
    wf = w.float().view(n_up // 128, 128, k // 128, 128)
    amax = wf.abs().amax(dim=(1, 3)).clamp_min(1e-4)
    inv = torch.full_like(amax, 448.0) / amax
    q = (wf * inv.view(n_up // 128, 1, k // 128, 1)).to(F8)
    s = amax / torch.full_like(amax, 448.0)
    return (q.double() * s.double().view(n_up // 128, 1, k // 128, 1)).view(n_up, k)[:n]


def _product(x, w, n):
    a = _deq_act(x)
    out = torch.empty(x.shape[0], n, dtype=torch.float64, device=x.device)
    for c in range(0, n, 8192):  # the 64-bit weights of the widest layer in pieces
        cols = min(8192, n - c)
        out[:, c:c + cols] = a @ _deq_w(w[c:c + (cols + 127) // 128 * 128], cols).t()
    return out


def exact(case, seed):
    op, k = case["op"], case["k"]
    i = _inputs(case, seed)
    x = i["x"]
    if op == "quantize":
        amax = x.double().view(case["m"], k // 128, 128).abs().amax(dim=2).clamp_min(1e-4)
        return (None, amax / 448.0)
    n = case["n"]
    if op == "decode_step":
        outs = []
        for j, xj in enumerate(x):
            up = _product(xj, i["w"][2 * j], n)
            outs += [up, _product(up.to(torch.bfloat16), i["w"][2 * j + 1], k)]
        return outs
    if op == "contiguous":
        out = torch.zeros(x.shape[0], n, dtype=torch.float64, device="cuda")
        r0 = 0
        for g, p in enumerate(i["padded"]):
            out[r0:r0 + p] = _product(x[r0:r0 + p], i["w"][g], n)
            r0 += p
        return out
    if op == "masked":
        g, m_max = case["groups"], case["m_max"]
        out = torch.zeros(g, m_max, n, dtype=torch.float64, device="cuda")
        for e, r in enumerate(i["rows"]):
            if r:
                out[e, :r] = _product(x[e * m_max:e * m_max + r], i["w"][e], n)
        return out
    d = _product(x, i["w"], n)
    if op == "gemm_e4m3":
        amax = d.view(case["m"], n // 128, 128).abs().amax(dim=2).clamp_min(1e-4)
        return (None, amax / 448.0)
    return d
