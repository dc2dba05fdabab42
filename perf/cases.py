"""What is timed on a B200: the work a user of this library has it do, through `llmmm_b200.capi`.

Five kinds of pass (`case["kind"]`):

  fp16_mm   one FP16 / BF16 GEMM (`fp16_mm`)
  fp8_mm    one FP8 blockwise GEMM, e4m3 output with fused 1x128 scales or fp32 output
  linears   the four projections of a transformer layer (qkv, o, gate_up, down), each on its own quantised
            activations with e4m3 output: the layer-shaped GEMM set without the fused hooks
  layer     the same projections chained as a serving program chains them: RMSNorm + quantise, qkv with q/k norm and
            rotary embedding fused, quantise the attention output, o projection to fp32, RMSNorm + quantise,
            gate_up with SwiGLU fused, down projection to fp32 (the attention itself is the caller's)
  mlp       gate_up and down of an MLP as plain GEMMs with e4m3 output
  weights   checkpoint weights made ready: [K, N] fp32 transposed, 128x128-quantised, and an e4m3 weight transposed

FP8 sources are N(0, 1) activations and N(0, 0.02) weights, FP16 / BF16 operands are uniform in [-1, 1): the
distributions the tests and the benchmark use.  Scratch is registered and weights are declared static once, in
`prepare`, as a serving program does.
"""
from __future__ import annotations

import math

import torch

from llmmm_b200 import capi

EPS = 1e-6
TABLE_ROWS = 8192  # rows of the rotary angle tables
# a drawn case costs no more than the largest listed one (the 7B-scale MLP below: 3.3e12 flops)
MAX_FLOPS = 3.3e12
MAX_BYTES = 2.0e9

# Qwen3-4B: hidden 2560, 32 query and 8 key / value heads of 128, intermediate 9728
QWEN3_4B = {"hidden": 2560, "q_heads": 32, "kv_heads": 8, "inter": 9728}


def listed():
    return [
        # the smallest call: launch and latency only (the first configuration of the benchmark's FP16 line)
        {"name": "fp16_256", "kind": "fp16_mm", "dtype": "float16", "M": 256, "N": 256, "K": 256},
        # the FP16 headline size
        {"name": "fp16_4096", "kind": "fp16_mm", "dtype": "float16", "M": 4096, "N": 4096, "K": 4096},
        # sizes that no tile divides, BF16: a caller with an odd number of rows and columns that are only 16-byte aligned
        {"name": "bf16_ragged", "kind": "fp16_mm", "dtype": "bfloat16", "M": 1001, "N": 2888, "K": 1544},
        # the FP8 headline size, output re-quantised in the epilogue
        {"name": "fp8_4096", "kind": "fp8_mm", "out": "e4m3", "M": 4096, "N": 4096, "K": 4096},
        # decode: one token of one request through a Qwen3-4B layer; weights dominate
        dict(QWEN3_4B, name="layer_m1", kind="layer", M=1),
        # decode: a batch of 16 requests
        dict(QWEN3_4B, name="layer_m16", kind="layer", M=16),
        # the largest decode batch of the weight-streaming path, plain projections
        dict(QWEN3_4B, name="linears_m64", kind="linears", M=64),
        # between decode and prefill, an odd number of rows
        dict(QWEN3_4B, name="linears_m100", kind="linears", M=100),
        # prefill of one prompt of odd length
        dict(QWEN3_4B, name="layer_m1333", kind="layer", M=1333),
        # prefill of a full chunk
        dict(QWEN3_4B, name="layer_m4096", kind="layer", M=4096),
        # 7B-scale MLP, large prefill batch: the largest
        {"name": "mlp7b_m8192", "kind": "mlp", "M": 8192, "hidden": 3584, "inter": 18944},
        # loading a checkpoint: the gate_up weight of a Qwen3-4B layer from fp32
        {"name": "weights_gate_up", "kind": "weights", "rows": 19456, "cols": 2560},
    ]


def _log(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(step, lo, int(round(v / step)) * step))


def _rows(rng):
    return _log(rng, 1, 8192)


def draw(rng):
    while True:
        kind = rng.choice(["fp16_mm", "fp8_mm", "linears", "layer", "layer", "mlp", "weights"])
        if kind == "fp16_mm":
            case = {"kind": kind, "dtype": rng.choice(["float16", "bfloat16"]), "M": _rows(rng), "N": _log(rng, 256, 12288, 8),
                    "K": _log(rng, 256, 12288, 8)}
        elif kind == "fp8_mm":
            case = {"kind": kind, "out": rng.choice(["e4m3", "f32"]), "M": _rows(rng), "N": _log(rng, 512, 38912, 128),
                    "K": _log(rng, 512, 18944, 128)}
        elif kind == "weights":
            case = {"kind": kind, "rows": _log(rng, 512, 38912, 128), "cols": _log(rng, 512, 18944, 128)}
        elif kind == "mlp":
            case = {"kind": kind, "M": _rows(rng), "hidden": _log(rng, 1024, 4096, 128), "inter": _log(rng, 2560, 18944, 128)}
        else:
            case = {"kind": kind, "M": _rows(rng), "hidden": _log(rng, 1024, 4096, 128), "q_heads": rng.choice([8, 16, 24, 28, 32]),
                    "kv_heads": rng.choice([2, 4, 8]), "inter": _log(rng, 2560, 14336, 128)}
        w = work(case)
        if w["flops"] <= MAX_FLOPS and w["bytes"] <= MAX_BYTES:
            return case


# ------------------------------------------------------------------ inputs ---

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(g, *shape, std=1.0):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32).mul_(std)


def _f32(*shape):
    return torch.zeros(*shape, device="cuda", dtype=torch.float32)


def _bytes(*shape):
    return torch.zeros(*shape, device="cuda", dtype=torch.uint8)


def _activations(g, M, K):
    """Quantised N(0, 1) activations: [M, K] e4m3 and [K/128, M] scales."""
    q, s = _bytes(M, K), _f32(K // 128, M)
    capi.fp8_quant_1x128(_normal(g, M, K), q, s, M, K)
    return q, s


def _weight(g, N, K):
    """A quantised N(0, 0.02) weight: [N, K] e4m3 and [N/128, K/128] scales."""
    q, s = _bytes(N, K), _f32(N // 128, K // 128)
    capi.fp8_quant_128x128(_normal(g, N, K, std=0.02), q, s, N, K)
    return q, s


def _quantised_out(M, N):
    return _bytes(M, N), _f32(N // 128, M)


def _shapes(case):
    """(N, K) of the projections of a layer."""
    H, I = case["hidden"], case["inter"]
    if case["kind"] == "mlp":
        return [(2 * I, H), (H, I)]
    q = case["q_heads"] * 128
    return [(q + 2 * case["kv_heads"] * 128, H), (H, q), (2 * I, H), (H, I)]


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    capi.set_static_weights(True)
    if kind == "fp16_mm":
        M, N, K = case["M"], case["N"], case["K"]
        dt = getattr(torch, case["dtype"])
        capi.ensure_workspace(max(M, 65), 256, 256)
        A = torch.rand(M, K, generator=g, device="cuda").mul_(2).sub_(1).to(dt)
        B = torch.rand(K, N, generator=g, device="cuda").mul_(2).sub_(1).to(dt)
        return dict(case, A=A, B=B, C=torch.zeros(M, N, device="cuda", dtype=dt))
    if kind == "fp8_mm":
        M, N, K = case["M"], case["N"], case["K"]
        capi.ensure_workspace(M, N, K)
        C = _quantised_out(M, N) if case["out"] == "e4m3" else (_f32(M, N),)
        return dict(case, A=_activations(g, M, K), B=_weight(g, N, K), C=C)
    if kind in ("linears", "mlp"):
        M, shapes = case["M"], _shapes(case)
        for N, K in shapes:
            capi.ensure_workspace(M, N, K)
        return dict(case, shapes=shapes, A=[_activations(g, M, K) for _, K in shapes], B=[_weight(g, N, K) for N, K in shapes],
                    C=[_quantised_out(M, N) for N, _ in shapes])
    if kind == "layer":
        M, H, I = case["M"], case["hidden"], case["inter"]
        shapes = _shapes(case)
        for N, K in shapes:
            capi.ensure_workspace(M, N, K)
        n_qkv, q = shapes[0][0], shapes[1][1]
        capi.ensure_qk_norm_rope_workspace(M, n_qkv, H)
        capi.ensure_swiglu_workspace(M, I, H)
        angle = torch.outer(torch.arange(TABLE_ROWS, device="cuda", dtype=torch.float32),
                            1e6 ** (-torch.arange(64, device="cuda", dtype=torch.float32) / 64))
        norm = lambda n: _normal(g, n, std=0.1).add_(1.0)  # noqa: E731
        return dict(case, x=_normal(g, M, H), attn=_normal(g, M, q), w_in=norm(H), w_post=norm(H), w_q=norm(128), w_k=norm(128),
                    cos=angle.cos().contiguous(), sin=angle.sin().contiguous(),
                    pos=torch.randint(0, TABLE_ROWS, (M,), generator=g, device="cuda", dtype=torch.int32),
                    n_qkv=n_qkv, q=q, B=[_weight(g, N, K) for N, K in shapes],
                    xq=_quantised_out(M, H), qkv=_quantised_out(M, n_qkv), aq=_quantised_out(M, q), o=_f32(M, H),
                    hq=_quantised_out(M, H), h=_quantised_out(M, I), y=_f32(M, H))
    R, C = case["rows"], case["cols"]  # weights: [C, R] in the checkpoint, [R, C] (output rows first) here
    return dict(case, w=_normal(g, C, R, std=0.02), q_t=torch.randint(0, 256, (C, R), generator=g, device="cuda", dtype=torch.uint8),
                wt=_f32(R, C), q=_bytes(R, C), s=_f32(R // 128, C // 128), q2=_bytes(R, C))


# -------------------------------------------------------------------- pass ---

def _e4m3(t):
    return t.view(torch.float8_e4m3fn)


def run(s):
    kind = s["kind"]
    if kind == "fp16_mm":
        capi.fp16_mm(s["A"], s["B"], s["C"], s["M"], s["N"], s["K"])
        return s["C"]
    if kind == "fp8_mm":
        (aq, as_), (bq, bs) = s["A"], s["B"]
        if s["out"] == "e4m3":
            capi.fp8_blockwise_mm(aq, as_, bq, bs, *s["C"], s["M"], s["N"], s["K"])
            return _e4m3(s["C"][0]), s["C"][1]
        capi.fp8_blockwise_mm_f32(aq, as_, bq, bs, s["C"][0], s["M"], s["N"], s["K"])
        return s["C"][0]
    if kind in ("linears", "mlp"):
        for (N, K), (aq, as_), (bq, bs), (cq, cs) in zip(s["shapes"], s["A"], s["B"], s["C"]):
            capi.fp8_blockwise_mm(aq, as_, bq, bs, cq, cs, s["M"], N, K)
        return [(_e4m3(cq), cs) for cq, cs in s["C"]]
    if kind == "layer":
        M, H, I, q = s["M"], s["hidden"], s["inter"], s["q"]
        qkv, o, gate_up, down = s["B"]
        capi.fp8_rmsnorm_quant_1x128(s["x"], s["w_in"], EPS, *s["xq"], M, H)
        capi.fp8_blockwise_mm_qk_norm_rope(*s["xq"], *qkv, *s["qkv"], s["pos"], s["cos"], s["sin"], s["w_q"], s["w_k"], EPS,
                                           s["q_heads"], s["kv_heads"], M, s["n_qkv"], H)
        capi.fp8_quant_1x128(s["attn"], *s["aq"], M, q)
        capi.fp8_blockwise_mm_f32(*s["aq"], *o, s["o"], M, H, q)
        capi.fp8_rmsnorm_quant_1x128(s["o"], s["w_post"], EPS, *s["hq"], M, H)
        capi.fp8_blockwise_mm_swiglu(*s["hq"], *gate_up, *s["h"], M, I, H)
        capi.fp8_blockwise_mm_f32(*s["h"], *down, s["y"], M, H, I)
        return {"qkv": (_e4m3(s["qkv"][0]), s["qkv"][1]), "o": s["o"], "h": (_e4m3(s["h"][0]), s["h"][1]), "y": s["y"]}
    R, C = s["rows"], s["cols"]
    capi.transpose_aligned_128(s["wt"], s["w"], C, R)
    capi.fp8_quant_128x128(s["wt"], s["q"], s["s"], R, C)
    capi.transpose_aligned_128(s["q2"], s["q_t"], C, R)
    return s["wt"], s["q"], s["s"], s["q2"]


# ------------------------------------------------------- work and tolerance ---

def _act_bytes(M, K):  # e4m3 and its 1x128 scales
    return M * K + 4 * M * K // 128


def _weight_bytes(N, K):
    return N * K + 4 * (N // 128) * (K // 128)


def work(case):
    kind = case["kind"]
    if kind == "weights":
        n = case["rows"] * case["cols"]
        # fp32 transposed, then quantised; an e4m3 weight transposed
        return {"bytes": (4 + 4) * n + (4 + 1) * n + 4 * n // 16384 + 2 * n, "flops": 0}
    M = case["M"]
    if kind == "fp16_mm":
        N, K = case["N"], case["K"]
        return {"bytes": 2 * (M * K + K * N + M * N), "flops": 2 * M * N * K}
    if kind == "fp8_mm":
        N, K = case["N"], case["K"]
        out = _act_bytes(M, N) if case["out"] == "e4m3" else 4 * M * N
        return {"bytes": _act_bytes(M, K) + _weight_bytes(N, K) + out, "flops": 2 * M * N * K}
    shapes = _shapes(case)
    flops = sum(2 * M * N * K for N, K in shapes)
    weights = sum(_weight_bytes(N, K) for N, K in shapes)
    if kind in ("linears", "mlp"):
        return {"bytes": weights + sum(_act_bytes(M, K) + _act_bytes(M, N) for N, K in shapes), "flops": flops}
    H, I, (n_qkv, _), (_, q) = case["hidden"], case["inter"], shapes[0], shapes[1]
    acts = 2 * (4 * M * H + 2 * _act_bytes(M, H))          # RMSNorm + quantise, read again by the projection, twice
    acts += _act_bytes(M, n_qkv) + 4 * M * 128 * 1         # qkv out; cos and sin rows
    acts += 4 * M * q + 2 * _act_bytes(M, q) + 4 * M * H   # attention output quantised and read; o out
    acts += 2 * _act_bytes(M, I) + 4 * M * H               # h out and read; y out
    return {"bytes": weights + acts, "flops": flops}


def tolerance(case):
    """Four times what the path differs by from itself with its sums in another order (tiles cut along K or not), and, for
    FP16 / BF16, from the fp64 product rounded once; the largest such difference seen stands beside each line."""
    kind = case["kind"]
    if kind == "weights":
        return "exact"  # copies and IEEE divisions
    if kind == "fp16_mm":
        # one rounding of an fp32 sum to 11 (8) bits: 5.4e-5 / 9.8e-4 for half, 1.5e-4 / 7.8e-3 for bfloat16
        return {"rel": 2.2e-4, "max": 4e-3} if case["dtype"] == "float16" else {"rel": 6e-4, "max": 0.032}
    if kind == "fp8_mm" and case["out"] == "f32":
        return {"rel": 1e-5, "max": 1e-4}
    # e4m3 results: a few values move by one step, which is 1/8 of the value at most: 2.0e-4
    if kind in ("fp8_mm", "linears", "mlp"):
        return {"rel": 8e-4, "max": 0.15}
    # chained, so that steps of the quantised intermediate values reach the outputs too: 1.7e-4
    return {"rel": 1e-3, "max": 0.15}


# ----------------------------------------------------------- 64-bit values ---

def _quant64(y, block_rows=1):
    """Values of the block quantisation as float64: (q, scale), block_rows x 128 blocks, q rounded to e4m3."""
    R, C = y.shape
    b = y.view(R // block_rows, block_rows, C // 128, 128)
    s = b.abs().amax(dim=(1, 3)) / 448.0
    q = torch.where(s[:, None, :, None] > 0, b / s[:, None, :, None], torch.zeros_like(b))
    return q.view(R, C).float().to(torch.float8_e4m3fn).double(), s


def _quant32(x, block_rows=1):
    """The quantised operands that `prepare` makes (IEEE fp32 divisions), de-quantised to float64."""
    R, C = x.shape
    b = x.view(R // block_rows, block_rows, C // 128, 128)
    s = b.abs().amax(dim=(1, 3), keepdim=True) / torch.tensor(448.0, device=x.device)
    q = torch.where(s > 0, b / s, torch.zeros_like(b)).to(torch.float8_e4m3fn)
    return (q.double() * s.double()).view(R, C)


def _out64(y):
    """(e4m3 values, [N/128, M] scales) of an e4m3 output."""
    q, s = _quant64(y)
    return q, s.t().contiguous()


def _deq64(y):
    q, s = _quant64(y)
    return q * s.repeat_interleave(128, dim=1)


def _rms64(x, w):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + EPS) * w


def exact(case, seed):
    kind = case["kind"]
    if kind == "weights":
        return None  # bytes: compared exactly
    g, M = _gen(seed), case["M"]
    if kind == "fp16_mm":
        dt = getattr(torch, case["dtype"])
        A = torch.rand(M, case["K"], generator=g, device="cuda").mul_(2).sub_(1).to(dt)
        B = torch.rand(case["K"], case["N"], generator=g, device="cuda").mul_(2).sub_(1).to(dt)
        return A.double() @ B.double()
    if kind == "fp8_mm":
        A = _quant32(_normal(g, M, case["K"]))
        B = _quant32(_normal(g, case["N"], case["K"], std=0.02), 128)
        return _out64(A @ B.t()) if case["out"] == "e4m3" else A @ B.t()
    shapes = _shapes(case)
    if kind in ("linears", "mlp"):
        A = [_quant32(_normal(g, M, K)) for _, K in shapes]
        B = [_quant32(_normal(g, N, K, std=0.02), 128) for N, K in shapes]
        return [_out64(a @ b.t()) for a, b in zip(A, B)]
    H, I, n_q, n_kv = case["hidden"], case["inter"], case["q_heads"], case["kv_heads"]
    x, attn = _normal(g, M, H).double(), _normal(g, M, n_q * 128)
    w_in, w_post, w_q, w_k = [_normal(g, n, std=0.1).add_(1.0).double() for n in (H, H, 128, 128)]
    angle = torch.outer(torch.arange(TABLE_ROWS, device="cuda", dtype=torch.float32),
                        1e6 ** (-torch.arange(64, device="cuda", dtype=torch.float32) / 64))
    pos = torch.randint(0, TABLE_ROWS, (M,), generator=g, device="cuda", dtype=torch.int32).long()
    cos, sin = angle.cos()[pos].double()[:, None], angle.sin()[pos].double()[:, None]
    w_qkv, w_o, w_gate_up, w_down = [_quant32(_normal(g, N, K, std=0.02), 128) for N, K in shapes]
    qkv = (_deq64(_rms64(x, w_in)) @ w_qkv.t()).view(M, -1, 128)
    for lo, hi, w in ((0, n_q, w_q), (n_q, n_q + n_kv, w_k)):
        h = _rms64(qkv[:, lo:hi], w)
        a, b = h[..., :64], h[..., 64:]
        qkv[:, lo:hi] = torch.cat([a * cos - b * sin, b * cos + a * sin], dim=2)
    o = _quant32(attn) @ w_o.t()
    acc = _deq64(_rms64(o, w_post)) @ w_gate_up.t()
    h = acc[:, :I] / (1 + torch.exp(-acc[:, :I])) * acc[:, I:]
    return {"qkv": _out64(qkv.reshape(M, -1)), "o": o, "h": _out64(h), "y": _deq64(h) @ w_down.t()}
