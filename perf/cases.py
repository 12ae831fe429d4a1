"""The workloads this library is timed on, on one GPU, through its public entry points (catccos_b200.capi, a thin
layer over the C ABI of include/catccos_b200.h).

A case is a dict of plain values:
  op     the entry point: "fused" (bf16 activations quantised on the fly, then the block-scaled matmul), "static" (the
         same without a symmetric buffer), "agmm" (activations that arrive quantised), "gemm" (the matmul on gathered
         operands), "gemm_quant" (its epilogue quantises the output for the next layer), "fp4" (FP4 quantiser, then the
         FP4 matmul), "quant" and "quant_ag" (the quantiser alone), "scatter" (the packed rows of an MoE dispatch)
  m n k  rows, output columns and contraction length (the quantisers have no n)
  codes  element type of the activations' codes: "e4m3" or "e5m2"
  out    element type of a matmul's result: "bf16" or "fp16"
  dist   distribution of the activations: "normal", or "outlier" (Student t with three degrees of freedom and 0.1 % of
         the channels a hundred times larger)
  top_k  destinations of a token ("scatter")
"""
import math

import torch

from catccos_b200 import capi

SYMM_BYTES = 1004 << 20  # what the reference's drivers reserve for their one symmetric buffer
STATIC_ELEMENTS = 8 << 20  # m * k of the allocation-free entry point
ACT_OPS = ("fused", "static", "fp4", "quant", "quant_ag", "scatter")  # these start from bf16 activations


def listed():
    return [
        # one decode step of 16 sequences through a tensor-parallel projection: weights stream, launches count
        dict(name="decode_fused", op="fused", m=16, n=4096, k=7168, codes="e4m3", out="bf16", dist="normal"),
        # the golden case of the reference's operator (256 rows, fp16 result): a small call
        dict(name="small_fused_fp16", op="fused", m=256, n=1024, k=1024, codes="e4m3", out="fp16", dist="normal"),
        # one rank's prefill chunk, the headline shape
        dict(name="prefill_fused", op="fused", m=1024, n=2304, k=7168, codes="e4m3", out="bf16", dist="normal"),
        # a long prefill with outlier channels
        dict(name="outlier_fused", op="fused", m=4096, n=3456, k=5120, codes="e4m3", out="bf16", dist="outlier"),
        # a latency-bound caller that may not allocate, with a batch that fits no tile
        dict(name="ragged_static", op="static", m=509, n=2320, k=3968, codes="e4m3", out="bf16", dist="normal"),
        # activations that arrive quantised to E5M2, ragged rows, the reference's output type
        dict(name="ragged_agmm_e5m2", op="agmm", m=3001, n=2064, k=5120, codes="e5m2", out="fp16", dist="normal"),
        # the gathered rows of eight ranks with 4096 rows each: the largest contraction
        dict(name="large_gemm", op="gemm", m=32768, n=3456, k=5120, codes="e4m3", out="bf16", dist="normal"),
        # a layer whose output feeds the next quantised layer
        dict(name="gemm_quant_out", op="gemm_quant", m=2048, n=7168, k=2304, codes="e4m3", out="bf16", dist="normal"),
        # FP4 activations and weights on the headline shape
        dict(name="prefill_fp4", op="fp4", m=1024, n=2304, k=7168, codes="e4m3", out="bf16", dist="normal"),
        # quantise-and-gather of one rank's prefill shard
        dict(name="quant_gather", op="quant_ag", m=4096, k=7168, codes="e4m3", dist="normal"),
        # a few ragged rows whose scale count is no multiple of four
        dict(name="quant_small_ragged", op="quant", m=37, k=1056, codes="e4m3", dist="normal"),
        # the dispatch side of a mixture-of-experts layer
        dict(name="moe_dispatch", op="scatter", m=2048, k=7168, top_k=8, codes="e4m3", dist="normal"),
    ]


# a drawn case costs no more than the largest listed one
MOST_FLOPS = 2.0 * 32768 * 3456 * 5120
MOST_BYTES = 2.0 * 32768 * 3456 + 1.04 * 5120 * (32768 + 3456)  # of the same call


def _spread(rng, low, high, step=1):
    """A multiple of `step` between the two, even over the logarithm."""
    v = math.exp(rng.uniform(math.log(low), math.log(high)))
    return min(high, max(low, int(round(v / step)) * step))


def draw(rng):
    while True:
        op = rng.choice(("fused", "fused", "static", "agmm", "gemm", "gemm_quant", "fp4", "quant", "quant_ag", "scatter"))
        c = dict(op=op, codes="e4m3", dist=rng.choice(("normal", "outlier")))
        if op == "scatter":
            c.update(m=_spread(rng, 16, 8192), k=_spread(rng, 1024, 7168, 32), top_k=rng.choice((1, 2, 4, 6, 8)))
        elif op in ("quant", "quant_ag"):
            c.update(m=_spread(rng, 16, 16384), k=_spread(rng, 512, 8192, 32), codes=rng.choice(("e4m3", "e4m3", "e5m2")))
        else:
            step_n = {"gemm_quant": 32, "fp4": 128}.get(op, 16)
            low, high = {"fused": (1, 8192), "static": (1, 4096), "agmm": (16, 16384), "gemm": (16, 32768), "gemm_quant": (16, 8192),
                         "fp4": (16, 8192)}[op]
            c.update(m=_spread(rng, low, high), n=_spread(rng, 1024, 7168, step_n), k=_spread(rng, 1024, 7168, 128),
                     out=rng.choice(("bf16", "fp16")))
            if op in ("fused", "static", "agmm", "gemm"):
                c["codes"] = rng.choice(("e4m3", "e4m3", "e5m2"))
        w = work(c)
        fits = op != "static" or c["m"] * c["k"] <= STATIC_ELEMENTS
        if fits and w["flops"] <= MOST_FLOPS and w["bytes"] <= MOST_BYTES:
            return c


def work(case):
    m, k = case["m"], case["k"]
    a16, a8, a4 = m * k * 2.0, m * k * (1.0 + 1.0 / 32), m * k * (0.5 + 1.0 / 32)
    if case["op"] in ("quant", "quant_ag"):
        return {"bytes": a16 + a8, "flops": 0.0}
    if case["op"] == "scatter":
        return {"bytes": a16 + m * case["top_k"] * (4.0 + capi.packed_row_bytes(k)), "flops": 0.0}
    n = case["n"]
    b8, b4 = n * k * (1.0 + 1.0 / 32), n * k * (0.5 + 1.0 / 32)
    c16, c8 = m * n * 2.0, m * n * (1.0 + 1.0 / 32)
    total = {"fused": a16 + b8 + c16, "static": a16 + b8 + c16, "agmm": a8 + b8 + c16, "gemm": a8 + b8 + c16,
             "gemm_quant": a8 + b8 + c8, "fp4": a16 + a4 + b4 + c16}[case["op"]]
    return {"bytes": total, "flops": 2.0 * m * n * k}


def tolerance(case):
    if case["op"] in ("quant", "quant_ag", "scatter"):
        return "exact"
    if case["op"] == "gemm_quant":
        # bytes; another order of the fp32 sums moves about one bf16 rounding in a thousand, and few of those move a code
        return {"rel": 0.0, "differ": 1e-3}
    # fp32 sums in another order, one rounding to 8 or 11 significant bits: at most one unit in the last place
    return {"rel": 4e-3, "max": 1.6e-2} if case["out"] == "bf16" else {"rel": 5e-4, "max": 2e-3}


_symm = None


def _symmetric_buffer():
    """One buffer for the whole process, as the reference's drivers allocate it."""
    global _symm
    if _symm is None:
        _symm = capi.symm_alloc(SYMM_BYTES)
    return _symm


def _activations(case, gen):
    m, k = case["m"], case["k"]
    x = torch.randn((m, k), generator=gen, device="cuda")
    if case["dist"] == "outlier":
        chi2 = torch.zeros_like(x)
        for _ in range(3):
            chi2 += torch.randn((m, k), generator=gen, device="cuda") ** 2
        x = x / (chi2 / 3.0).clamp_min(1e-6).sqrt()
        x[:, torch.randperm(k, generator=gen, device="cuda")[: math.ceil(0.001 * k)]] *= 100.0
    return x.to(torch.bfloat16)


EMAX = {"e4m3": 8, "e5m2": 15, "e2m1": 2}


def _mx_rows(x, codes):
    """MX-quantises bf16 [rows, k] along k: codes (uint8 [rows, k], or [rows, k / 2] for "e2m1") and E8M0 scales."""
    rows, k = x.shape
    block = x.float().view(rows, k // 32, 32)
    exponent = torch.frexp(block.abs().amax(dim=2).clamp_min(1e-12))[1] - 1 - EMAX[codes]
    scaled = torch.ldexp(block, -exponent.unsqueeze(2)).view(rows, k)
    scales = (exponent + 127).to(torch.uint8)
    if codes == "e2m1":
        edges = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=x.device)
        q = torch.bucketize(scaled.abs(), edges).to(torch.uint8) | (torch.signbit(scaled).to(torch.uint8) << 3)
        return q[:, 0::2] | (q[:, 1::2] << 4), scales
    most, dtype = (448.0, torch.float8_e4m3fn) if codes == "e4m3" else (57344.0, torch.float8_e5m2)
    return scaled.clamp(-most, most).to(dtype).view(torch.uint8), scales


def _weights(case, gen, codes):
    """N(0, 0.02) quantised along k: codes [k, n] (FP4: two columns to a byte) and scales [k / 64, n, 2]."""
    n, k = case["n"], case["k"]
    w = (torch.randn((n, k), generator=gen, device="cuda") * 0.02).to(torch.bfloat16)
    q, s = _mx_rows(w, codes)
    if codes == "e2m1":
        values = torch.stack((q & 15, q >> 4), dim=2).view(n, k).t()
        q = (values[:, 0::2] | (values[:, 1::2] << 4)).contiguous()
    else:
        q = q.t().contiguous()
    return q, s.view(n, k // 64, 2).permute(1, 0, 2).contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    op, m, k = case["op"], case["m"], case["k"]
    # element types are the library's options, set once by a program that serves one model
    capi.set_option("a_dtype", 1 if case["codes"] == "e5m2" else 0)
    capi.set_option("b_dtype", 0)
    capi.set_option("c_dtype", 1 if case.get("out") == "fp16" else 0)
    s = {"op": op, "symm": _symmetric_buffer()}
    x = _activations(case, gen)
    if op in ACT_OPS:
        s["x"] = x
    else:
        s["a"], s["a_scales"] = _mx_rows(x, case["codes"])
    if "n" in case:
        s["b"], s["b_scales"] = _weights(case, gen, "e2m1" if op == "fp4" else "e4m3")
        s["c"] = torch.zeros((m, case["n"]), dtype=torch.float16 if case["out"] == "fp16" else torch.bfloat16, device="cuda")
    if op == "quant_ag":
        s["codes"] = torch.zeros((m, k), dtype=torch.uint8, device="cuda")
        s["scales"] = torch.zeros((m, k // 32), dtype=torch.uint8, device="cuda")
    if op == "scatter":
        # every token's rows are scattered over the expert buffers; a few routes are dropped, their rows stay as they are
        rows = m * case["top_k"]
        index = torch.randperm(rows, generator=gen, device="cuda").to(torch.int32)
        index[torch.rand(rows, generator=gen, device="cuda") < 0.02] = -1
        s["index"], s["top_k"] = index.view(m, case["top_k"]).contiguous(), case["top_k"]
        s["packed"] = torch.zeros((rows, capi.packed_row_bytes(k)), dtype=torch.uint8, device="cuda")
    return s


def run(s):
    op = s["op"]
    if op == "fused":
        capi.mx_quant_allgather_matmul(s["x"], s["b"], s["b_scales"], s["c"], s["symm"], 1)
        return s["c"]
    if op == "static":
        capi.mx_quant_matmul_static(s["x"], s["b"], s["b_scales"], s["c"])
        return s["c"]
    if op == "agmm":
        capi.fp8_mx_allgather_matmul(s["a"], s["a_scales"], s["b"], s["b_scales"], s["c"], s["symm"], 1)
        return s["c"]
    if op == "gemm":
        return capi.mx_gemm(s["a"], s["a_scales"], s["b"], s["b_scales"], out=s["c"])
    if op == "gemm_quant":
        return capi.mx_gemm_quant_out(s["a"], s["a_scales"], s["b"], s["b_scales"])
    if op == "fp4":
        packed, scales = capi.mx_quant_fp4(s["x"])
        capi.fp4_mx_allgather_matmul(packed, scales, s["b"], s["b_scales"], s["c"], s["symm"], 1)
        return packed, scales, s["c"]
    if op == "quant":
        return capi.mx_quant(s["x"])
    if op == "quant_ag":
        capi.mx_quant_allgather(s["x"], s["codes"], s["scales"], s["symm"], 1)
        return s["codes"], s["scales"]
    capi.mx_quant_scatter_packed(s["x"], s["index"], s["packed"], s["top_k"])
    return s["packed"]
