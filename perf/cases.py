"""The work that this library is measured by, called through its public entry points.

Four kinds of case, one per family of entry points:

  attn     ops.fa_fwd        attention forward, bf16 [B, H, S, D]
  gemm     ops.gemm          C = A B, bf16 operands, bf16 or fp32 out
  grouped  ops.gemm_grouped  G products of one shape
  rowwise  ops.softmax / ops.layer_norm, or ops.rms_norm followed by ops.swiglu, fp32

`listed()` names the fixed cases, `draw()` gives more of the same ranges: sequence lengths of
128 to 8192 (odd ones too), both head dims, causal and not, grouped K/V heads, with and
without the log-sum-exp; products from one tile to 8192 cubed; groups of 2 to 64; rows of
256 to 32768 columns, 16 to 65536 of them.
"""
from __future__ import annotations

import math

import torch

import __graft_entry__

ops = __graft_entry__.load_package().ops


def _attn(name, B, H, H_kv, S, D, causal, lse=False, sigma=1.0):
    return {"name": name, "kind": "attn", "B": B, "H": H, "H_kv": H_kv, "S": S, "D": D, "causal": causal, "lse": lse,
            "sigma": sigma}


def listed():
    return [
        # one short prompt on few heads: the correctness check of the attention driver, all latency
        _attn("attn_short_prompt", 1, 2, 2, 512, 128, False),
        # one long prompt being prefilled: grouped K/V heads, a length that is no multiple of
        # anything, the log-sum-exp kept for the backward pass or for merging with other keys
        _attn("attn_prefill_gqa_lse", 1, 32, 8, 3001, 128, True, lse=True),
        # an encoder batch, the headline benchmark
        _attn("attn_d128", 4, 16, 16, 4096, 128, False),
        # many short sequences with small heads, the benchmark's second configuration
        _attn("attn_d64", 16, 16, 16, 2048, 64, False),
        # a training batch with long causal sequences, the benchmark's third configuration
        _attn("attn_causal_long", 8, 32, 32, 8192, 128, True, sigma=0.5),
        # a few tokens against a square weight matrix: few output tiles, the weights' bytes count
        {"name": "gemm_few_rows", "kind": "gemm", "M": 128, "N": 4096, "K": 4096, "f32_out": False},
        # a deep product with a small result kept in fp32, as for a weight gradient
        {"name": "gemm_deep_f32", "kind": "gemm", "M": 1024, "N": 1152, "K": 8192, "f32_out": True},
        # the benchmark's dense product
        {"name": "gemm_square", "kind": "gemm", "M": 8192, "N": 8192, "K": 8192, "f32_out": False},
        # many small problems of one shape, as experts or heads make them
        {"name": "grouped_gemm", "kind": "grouped", "G": 64, "M": 256, "N": 1024, "K": 1024, "f32_out": False},
        # a handful of tokens through a norm: one small launch
        {"name": "layer_norm_few_rows", "kind": "rowwise", "op": "layer_norm", "rows": 16, "N": 2048},
        # scores over a long axis, a few thousand rows
        {"name": "softmax_long_rows", "kind": "rowwise", "op": "softmax", "rows": 4096, "N": 30000},
        # the row-wise work around a feed-forward block for a whole batch: norm in, gate in the middle
        {"name": "rms_norm_swiglu", "kind": "rowwise", "op": "rms_norm_swiglu", "rows": 16384, "N": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["attn", "gemm", "grouped", "rowwise"], [0.45, 0.25, 0.1, 0.2])[0]
    if kind == "attn":
        while True:
            D = rng.choice([64, 128])
            causal = rng.random() < 0.5
            S = _log_int(rng, 128, 8192)
            if rng.random() < 0.5:
                S = (S + 63) // 128 * 128
            H_kv = rng.choice([1, 2, 4, 8, 12, 16, 32])
            H = H_kv * rng.choice([1, 1, 2, 4])
            B = _log_int(rng, 1, 64)
            # the tiles above the diagonal of a short causal problem count as work here
            if 4.0 * B * H * S * S * D <= 2.5e12 and B * H * S <= 1 << 21:
                return {"kind": "attn", "B": B, "H": H, "H_kv": H_kv, "S": S, "D": D, "causal": causal,
                        "lse": rng.random() < 0.3, "sigma": rng.choice([0.5, 1.0])}
    if kind == "gemm":
        return {"kind": "gemm", "M": 128 * _log_int(rng, 1, 64), "N": 128 * _log_int(rng, 1, 64),
                "K": 64 * _log_int(rng, 2, 128), "f32_out": rng.random() < 0.4}
    if kind == "grouped":
        return {"kind": "grouped", "G": _log_int(rng, 2, 64), "M": 128 * _log_int(rng, 1, 8),
                "N": 64 * _log_int(rng, 1, 32), "K": 64 * _log_int(rng, 1, 32), "f32_out": rng.random() < 0.4}
    op = rng.choice(["softmax", "layer_norm", "rms_norm_swiglu"])
    N = 4 * _log_int(rng, 64, 8192)
    rows = _log_int(rng, 16, min(65536, (1 << 27) // N))
    return {"kind": "rowwise", "op": op, "rows": rows, "N": N}


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    kind = case["kind"]
    state = dict(case)
    if kind == "attn":
        B, H, H_kv, S, D = (case[k] for k in ("B", "H", "H_kv", "S", "D"))

        def normal(heads, sigma):
            return torch.randn(B, heads, S, D, device=dev, generator=g).mul_(sigma).to(torch.bfloat16)

        state["q"], state["k"], state["v"] = normal(H, case["sigma"]), normal(H_kv, case["sigma"]), normal(H_kv, 1.0)
        state["lse_out"] = torch.empty(B, H, S, device=dev) if case["lse"] else None
    elif kind in ("gemm", "grouped"):
        lead = (case["G"],) if kind == "grouped" else ()

        def uniform(rows):
            return torch.rand(*lead, rows, case["K"], device=dev, generator=g).mul_(2).sub_(1).to(torch.bfloat16)

        state["a"], state["bt"] = uniform(case["M"]), uniform(case["N"])
    else:
        rows, N = case["rows"], case["N"]
        state["x"] = torch.randn(rows, N, device=dev, generator=g)
        state["w"] = torch.randn(N, device=dev, generator=g).mul_(0.1).add_(1.0)
        state["bias"] = torch.randn(N, device=dev, generator=g).mul_(0.1)
        if case["op"] == "rms_norm_swiglu":
            state["gate"] = torch.randn(rows, N, device=dev, generator=g)
            state["up"] = torch.randn(rows, N, device=dev, generator=g)
    return state


def run(state):
    kind = state["kind"]
    if kind == "attn":
        o = ops.fa_fwd(state["q"], state["k"], state["v"], causal=state["causal"], lse=state["lse_out"])
        return [o] if state["lse_out"] is None else [o, state["lse_out"]]
    if kind == "gemm":
        return ops.gemm(state["a"], state["bt"], f32_out=state["f32_out"])
    if kind == "grouped":
        return ops.gemm_grouped(state["a"], state["bt"], f32_out=state["f32_out"])
    if state["op"] == "softmax":
        return ops.softmax(state["x"])
    if state["op"] == "layer_norm":
        return ops.layer_norm(state["x"], state["w"], state["bias"])
    return [ops.rms_norm(state["x"], state["w"]), ops.swiglu(state["gate"], state["up"])]


def work(case):
    kind = case["kind"]
    if kind == "attn":
        B, H, H_kv, S, D = (case[k] for k in ("B", "H", "H_kv", "S", "D"))
        pairs = S * (S + 1) // 2 if case["causal"] else S * S   # (query, key) pairs of one head
        return {"bytes": 2 * B * S * D * (2 * H + 2 * H_kv) + (4 * B * H * S if case["lse"] else 0),
                "flops": 4 * B * H * D * pairs}
    if kind in ("gemm", "grouped"):
        G, M, N, K = case.get("G", 1), case["M"], case["N"], case["K"]
        return {"bytes": G * (2 * K * (M + N) + M * N * (4 if case["f32_out"] else 2)), "flops": 2 * G * M * N * K}
    n = case["rows"] * case["N"]
    # bytes: each matrix once in, once out; flops: a few per element, far from mattering
    return {"bytes": 4 * n * (5 if case["op"] == "rms_norm_swiglu" else 2), "flops": 5 * n}


def exact(case, seed):
    """What run() returns on prepare(case, seed), in 64 bits with torch's own operations."""
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "attn":
        return _attn_exact(case, s["q"], s["k"], s["v"])
    if kind in ("gemm", "grouped"):
        return s["a"].double() @ s["bt"].double().mT
    x, w = s["x"].double(), s["w"].double()
    if case["op"] == "softmax":
        return torch.softmax(x, dim=1)
    if case["op"] == "layer_norm":
        y = x - x.mean(dim=1, keepdim=True)
        return y * torch.rsqrt(y.square().mean(dim=1, keepdim=True) + 1e-5) * w + s["bias"].double()
    y = x * torch.rsqrt(x.square().mean(dim=1, keepdim=True) + 1e-6) * w
    gate = s["gate"].double()
    return [y, gate * torch.sigmoid(gate) * s["up"].double()]


def _attn_exact(case, q, k, v):
    B, H, S, D = q.shape
    group = H // case["H_kv"]
    o = torch.empty(B, H, S, D, device=q.device, dtype=torch.float64)
    lse = torch.empty(B, H, S, device=q.device, dtype=torch.float64)
    rows = 4096                              # query rows of one head at a time: 0.27 GB of scores at most
    keys = torch.arange(S, device=q.device)
    for b in range(B):
        for h in range(H):
            kd, vd = k[b, h // group].double(), v[b, h // group].double()
            for r in range(0, S, rows):
                scores = q[b, h, r:r + rows].double() @ kd.mT
                scores *= D ** -0.5
                if case["causal"]:
                    scores.masked_fill_(keys[None, :] > keys[r:r + rows, None], -math.inf)
                top = scores.amax(dim=1, keepdim=True)
                scores.sub_(top).exp_()
                total = scores.sum(dim=1, keepdim=True)
                o[b, h, r:r + rows] = (scores @ vd) / total
                lse[b, h, r:r + rows] = (top + total.log())[:, 0]
    return [o, lse] if case["lse"] else [o]


def tolerance(case):
    """Four to seven times the distance to the same result computed in 64 bits, which each line gives."""
    kind = case["kind"]
    if kind == "attn":
        # P and O are bf16: 2.0e-3 to 2.4e-3 at every size, causal or not (log-sum-exp: 4e-7)
        return {"rel": 1e-2}
    if kind in ("gemm", "grouped"):
        # fp32 sums: 4e-7 (K = 512) to 1.9e-6 (K = 8192); bf16 out: one rounding, 1.7e-3
        return {"rel": 1e-5} if case["f32_out"] else {"rel": 7e-3}
    # fp32 in and out: 5e-8 to 7e-8 (norms and gate), 1.4e-7 (softmax, hardware exponentials)
    return {"rel": 1e-6}
