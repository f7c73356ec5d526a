"""The quantized linear layers that a program built on `hipkittens` runs, as measured cases.

One pass is what such a program does for one batch of activations: the activations (bf16, new each time) are quantized by one
public call and multiplied with weights that were quantized once, by a second one.  Kinds of layer:

  pts        per-token FP8 (optionally batched, with bias)
  blockscale 1x128 / 128x128 block-scaled FP8; `rms`: the quantizer's fused RMSNorm; `mul_add`: the fused C = c_a * gemm + c_b
  mxfp4      MXFP4; `tc`: scale factors kept in the tensor core's layout, else row-major ones as the reference project passes them
  ptgq       bf16 activations re-quantized per 64 K elements inside the GEMM, one scale per weight tensor
  moe_fp8    grouped block-scaled FP8 GEMM over expert-sorted rows
  moe_mxfp4  grouped MXFP4 GEMM over a padded, expert-sorted row list

Sizes are those of the repository's benchmark configurations and tests: M from a single decoded token to a 16384-row prefill,
N to 57344, K to 8192, row counts that are not multiples of any tile, N that is only a multiple of 8 where the layer takes it.
"""
import os
import sys

import torch

_PACKAGE = os.path.abspath("amd-kernels_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)
import hipkittens as hk  # noqa: E402

DEV = "cuda"
EPS = 1e-6


def listed():
    return [
        # The smallest layer of the benchmark: launches and host calls are most of it.
        {"name": "pts_small", "kind": "pts", "batch": 1, "M": 128, "N": 1024, "K": 1024, "bias": False},
        # One decode step of 16 sequences through a large projection: the weights have to cross HBM once.
        {"name": "pts_decode", "kind": "pts", "batch": 1, "M": 16, "N": 28672, "K": 8192, "bias": False},
        # Eight independent projections of 512 rows with bias.
        {"name": "pts_batched", "kind": "pts", "batch": 8, "M": 512, "N": 4096, "K": 4096, "bias": True},
        # A decode step of a block-scaled MLP up-projection behind its RMSNorm, a batch that fills no tile.
        {"name": "block_decode", "kind": "blockscale", "M": 24, "N": 14336, "K": 4096, "rms": True, "mul_add": False},
        # The same layer in prefill.
        {"name": "block_prefill", "kind": "blockscale", "M": 4096, "N": 14336, "K": 4096, "rms": True, "mul_add": False},
        # The largest layer that the benchmark runs on one GPU.
        {"name": "block_largest", "kind": "blockscale", "M": 16384, "N": 57344, "K": 8192, "rms": False, "mul_add": False},
        # Decode with MXFP4 weights whose scale factors were laid out once when they were loaded.
        {"name": "fp4_decode", "kind": "mxfp4", "M": 16, "N": 28672, "K": 8192, "tc": True, "mul_add": False},
        # MXFP4 prefill.
        {"name": "fp4_prefill", "kind": "mxfp4", "M": 8192, "N": 8192, "K": 8192, "tc": True, "mul_add": False},
        # The reference project's own call (row-major scale factors) on a mid-sized ragged problem, with the fused multiply-add.
        {"name": "fp4_ragged", "kind": "mxfp4", "M": 1000, "N": 3080, "K": 4224, "tc": False, "mul_add": True},
        # In-loop re-quantization: four ragged batches with bias.
        {"name": "ptgq_batched", "kind": "ptgq", "batch": 4, "M": 500, "N": 4096, "K": 4096, "bias": True},
        # A prefill through a mixture of experts: 8192 tokens, top-2 of 8 experts.
        {"name": "moe_fp8_prefill", "kind": "moe_fp8", "tokens": 8192, "experts": 8, "top_k": 2, "N": 14336, "K": 4096, "bias": False},
        # A decode step of 64 sequences through a mixture of MXFP4 experts.
        {"name": "moe_fp4_decode", "kind": "moe_mxfp4", "tokens": 64, "experts": 8, "top_k": 2, "N": 8192, "K": 8192},
    ]


def draw(rng):
    def size(low, high, multiple):
        """Log-uniform over [low, high], a multiple of `multiple`."""
        v = low * (high / low) ** rng.random()
        return max(multiple, int(round(v / multiple)) * multiple)

    def rows(high):
        """Log-uniform row counts; most are not multiples of anything."""
        return size(1, high, 1)

    def cols():
        """Mostly whole 128-column blocks, one in four ragged."""
        return size(1024, 28672, 128 if rng.random() < 0.75 else 8)

    kind = rng.choice(["pts", "pts", "blockscale", "blockscale", "mxfp4", "mxfp4", "ptgq", "moe_fp8", "moe_mxfp4"])
    if kind == "pts":
        batch = rng.choice([1, 1, 1, 2, 4, 8])
        if batch == 1:
            return {"kind": kind, "batch": 1, "M": rows(8192), "N": cols(), "K": size(1024, 8192, 128), "bias": False}
        return {"kind": kind, "batch": batch, "M": size(16, 1024, 1), "N": size(1024, 4096, 8), "K": size(1024, 4096, 128), "bias": rng.random() < 0.5}
    if kind == "blockscale":
        return {"kind": kind, "M": rows(8192), "N": size(1024, 57344, 128), "K": size(1024, 8192, 128), "rms": rng.random() < 0.5,
                "mul_add": rng.random() < 0.25}
    if kind == "mxfp4":
        return {"kind": kind, "M": rows(8192), "N": cols(), "K": size(1024, 8192, 128), "tc": rng.random() < 0.5, "mul_add": False}
    if kind == "ptgq":
        return {"kind": kind, "batch": rng.choice([1, 2, 4]), "M": rows(2048), "N": size(1024, 8192, 8), "K": size(1024, 4096, 64),
                "bias": rng.random() < 0.5}
    experts = rng.choice([8, 16])
    case = {"kind": kind, "tokens": rows(8192), "experts": experts, "top_k": rng.choice([2, 4]), "N": size(1024, 8192, 128),
            "K": size(1024, 4096, 128)}
    if kind == "moe_fp8":
        case["bias"] = rng.random() < 0.5
    return case


# ---- inputs ---------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _activations(g, rows, K):
    """N(0, 1) with 1 % of the channels 20 times as large (outlier channels)."""
    x = torch.randn(rows, K, generator=g, device=DEV)
    x[:, torch.randperm(K, generator=g, device=DEV)[: max(1, K // 100)]] *= 20.0
    return x.bfloat16()


def _weights(g, N, K):
    return (torch.randn(N, K, generator=g, device=DEV) * 0.02).bfloat16()


def _empty(*shape, dtype=torch.bfloat16):
    return torch.empty(*shape, dtype=dtype, device=DEV)


def _zeros(*shape, dtype=torch.uint8):
    return torch.zeros(*shape, dtype=dtype, device=DEV)


def _routing(g, tokens, experts, top_k):
    """Random top-k routing: experts of every flat (token, k) index, the stable order by expert, rows per expert."""
    picks = torch.rand(tokens, experts, generator=g, device=DEV).topk(top_k, dim=1).indices.reshape(-1)
    return picks, torch.argsort(picks, stable=True).int(), torch.bincount(picks, minlength=experts).tolist()


def _prepare_pts(c, g):
    B, M, N, K = c["batch"], c["M"], c["N"], c["K"]
    s = {"x": _activations(g, B * M, K), "xq": _empty(B * M, K, dtype=torch.uint8), "xs": _empty(B * M, 1, dtype=torch.float32),
         "wq": _empty(B * N, K, dtype=torch.uint8), "ws": _empty(B * N, 1, dtype=torch.float32), "bias": None}
    hk.per_token_quant_fwd(_weights(g, B * N, K), s["wq"], s["ws"])
    if B == 1:
        s["y"] = _empty(M, N)
    else:
        s["y"] = _empty(B, M, N)
        s["xq3"], s["wq3"] = s["xq"].view(B, M, K), s["wq"].view(B, N, K)
        if c["bias"]:
            s["bias"] = torch.randn(B, N, generator=g, device=DEV).bfloat16()
    return s


def _run_pts(c, s):
    hk.per_token_quant_fwd(s["x"], s["xq"], s["xs"])
    if c["batch"] == 1:
        hk.gemm.a8w8_per_token.dispatch(s["xq"], s["wq"], s["y"], s["xs"], s["ws"])
    else:
        hk.batched_gemm.a8w8.dispatch(s["xq3"], s["wq3"], s["xs"], s["ws"], s["y"], s["bias"])
    return s["y"], s["xq"], s["xs"]


def _prepare_blockscale(c, g):
    M, N, K = c["M"], c["N"], c["K"]
    s = {"x": _activations(g, M, K), "xq": _empty(M, K, dtype=torch.uint8), "xs": _empty(M, K // 128, dtype=torch.float32),
         "wq": _empty(N, K, dtype=torch.uint8), "ws": _empty(K // 128, N // 128, dtype=torch.float32), "y": _empty(M, N), "norm": None}
    hk.weight_quant_128x128(_weights(g, N, K), s["wq"], s["ws"])
    if c["rms"]:
        s["norm"] = (1.0 + 0.1 * torch.randn(K, generator=g, device=DEV)).bfloat16()
    if c["mul_add"]:
        s["c_a"], s["c_b"] = torch.randn(2, M, N, generator=g, device=DEV).bfloat16().unbind(0)
    return s


def _run_blockscale(c, s):
    hk.fused_rmsnorm_fp8_quant_fwd(s["x"], s["norm"], s["xq"], s["xs"], EPS)
    if c["mul_add"]:
        hk.fused_gemm.a8w8_blockscale_mul_add.dispatch(s["xq"], s["wq"], s["y"], s["xs"], s["ws"], s["c_a"], s["c_b"])
    else:
        hk.gemm.a8w8_blockscale.dispatch(s["xq"], s["wq"], s["y"], s["xs"], s["ws"])
    return s["y"], s["xq"], s["xs"]


def _prepare_mxfp4(c, g):
    M, N, K = c["M"], c["N"], c["K"]
    s = {"x": _activations(g, M, K), "xq": _empty(M, K // 2, dtype=torch.uint8), "wq": _empty(N, K // 2, dtype=torch.uint8), "y": _empty(M, N)}
    ws = _empty(N, K // 32, dtype=torch.uint8)
    hk.fused_rmsnorm_mxfp4_quant_fwd(_weights(g, N, K), None, s["wq"], ws, EPS)
    if c["tc"]:
        s["xs"] = _zeros(hk.gemm.afp4wfp4.sf_tc_bytes(1, M, K))
        s["ws"] = _zeros(hk.gemm.afp4wfp4.sf_tc_bytes(1, N, K))
        hk.gemm.afp4wfp4.sf_to_tc(ws, s["ws"], K)
    else:
        s["xs"], s["ws"] = _empty(M, K // 32, dtype=torch.uint8), ws
    if c["mul_add"]:
        s["c_a"], s["c_b"] = torch.randn(2, M, N, generator=g, device=DEV).bfloat16().unbind(0)
    return s


def _run_mxfp4(c, s):
    if c["tc"]:
        hk.fused_rmsnorm_mxfp4_quant_tc_fwd(s["x"], None, s["xq"], None, s["xs"], EPS)
        hk.gemm.afp4wfp4.dispatch_tc(s["xq"], s["wq"], s["y"], s["xs"], s["ws"], True, True)
    else:
        hk.fused_rmsnorm_mxfp4_quant_fwd(s["x"], None, s["xq"], s["xs"], EPS)
        if c["mul_add"]:
            hk.fused_gemm.afp4wfp4_mul_add.dispatch(s["xq"], s["wq"], s["y"], s["xs"], s["ws"], s["c_a"], s["c_b"])
        else:
            hk.gemm.afp4wfp4.dispatch(s["xq"], s["wq"], s["y"], s["xs"], s["ws"])
    return s["y"], s["xq"], s["xs"]


def _prepare_ptgq(c, g):
    B, M, N, K = c["batch"], c["M"], c["N"], c["K"]
    w = _weights(g, B * N, K)
    s = {"x": _activations(g, B * M, K).view(B, M, K), "wq": _empty(B, N, K, dtype=torch.uint8), "y": _empty(B, M, N), "bias": None}
    s["ws"] = (w.abs().max().float() / 448.0).reshape(1)
    hk.moe_routing.quant.downcast_to_static_fp8(w, s["wq"], s["ws"], B * N, K)
    if c["bias"]:
        s["bias"] = torch.randn(B, 1, N, generator=g, device=DEV).bfloat16()
    return s


def _run_ptgq(c, s):
    hk.batched_gemm.a8w8_ptgq.dispatch(s["x"], s["wq"], s["ws"], s["y"], s["bias"])
    return s["y"]


def _prepare_moe_fp8(c, g):
    T, E, N, K = c["tokens"], c["experts"], c["N"], c["K"]
    rows = T * c["top_k"]
    _, order, hist = _routing(g, T, E, c["top_k"])
    tiles = [e | (b << 16) for e in range(E) for b in range((hist[e] + 127) // 128)]
    offs = [sum(hist[:e]) for e in range(E)]
    s = {"x": _activations(g, T, K), "xq": _empty(T, K, dtype=torch.uint8), "xs": _empty(T, K // 128, dtype=torch.float32),
         "wq": _empty(E, N, K, dtype=torch.uint8), "ws": _empty(E, K // 128, N // 128, dtype=torch.float32), "y": _empty(rows, N),
         "gather": order, "hist": torch.tensor(hist, dtype=torch.int32, device=DEV), "offs": torch.tensor(offs, dtype=torch.int32, device=DEV),
         "tiles": torch.tensor(tiles, dtype=torch.int32, device=DEV), "bias": None}
    for e in range(E):
        hk.weight_quant_128x128(_weights(g, N, K), s["wq"][e], s["ws"][e])
    s["w_view"] = s["wq"].transpose(1, 2)
    if c["bias"]:
        s["bias"] = torch.randn(E, N, generator=g, device=DEV)
    return s


def _run_moe_fp8(c, s):
    N, K = c["N"], c["K"]
    kb, nb = K // 128, N // 128
    hk.fused_rmsnorm_fp8_quant_fwd(s["x"], None, s["xq"], s["xs"], EPS)
    hk.moe_gemm.a8w8_blockscale.moe_a8w8_blockscale(
        s["xq"], s["w_view"], s["y"], s["xs"], s["ws"], s["bias"], s["gather"], s["hist"], s["offs"], s["tiles"], N, K, 128, 128,
        s["tiles"].numel(), nb, c["top_k"], N, 1, K, 1, N * K, 1, K, kb, 1, kb * nb, nb, 1)
    return s["y"], s["xq"], s["xs"]


def _prepare_moe_mxfp4(c, g):
    T, E, N, K = c["tokens"], c["experts"], c["N"], c["K"]
    rows = T * c["top_k"]
    _, order, hist = _routing(g, T, E, c["top_k"])
    ids, experts, at = [], [], 0
    for e in range(E):
        pad = -hist[e] % 128
        ids += [order[at: at + hist[e]], torch.full((pad,), rows, dtype=torch.int32, device=DEV)]
        experts += [e] * ((hist[e] + pad) // 128)
        at += hist[e]
    s = {"x": _activations(g, T, K), "xq": _empty(T, K // 2, dtype=torch.uint8), "xs": _empty(T, K // 32, dtype=torch.uint8),
         "wq": _empty(E, N, K // 2, dtype=torch.uint8), "ws": _empty(E, N, K // 32, dtype=torch.uint8), "y": _empty(rows, N),
         "ids": torch.cat(ids), "experts": torch.tensor(experts, dtype=torch.int32, device=DEV),
         "gate": torch.rand(rows, generator=g, device=DEV)}
    for e in range(E):
        hk.fused_rmsnorm_mxfp4_quant_fwd(_weights(g, N, K), None, s["wq"][e], s["ws"][e], EPS)
    s["w_view"], s["ws_view"] = s["wq"].transpose(1, 2), s["ws"].transpose(1, 2)
    return s


def _run_moe_mxfp4(c, s):
    N, K = c["N"], c["K"]
    hk.fused_rmsnorm_mxfp4_quant_fwd(s["x"], None, s["xq"], s["xs"], EPS)
    hk.moe_gemm.mxfp4.moe_mxfp4(
        s["xq"], s["w_view"], s["y"], s["xs"], s["ws_view"], None, None, s["gate"], s["ids"], s["experts"], N, K, c["tokens"] * c["top_k"],
        c["top_k"], True, K // 2, 1, N * K // 2, 1, K // 2, N, 1, K // 32, 1, N * K // 32, 1, K // 32, s["experts"].numel(), N // 128)
    return s["y"], s["xq"], s["xs"]


_KINDS = {"pts": (_prepare_pts, _run_pts), "blockscale": (_prepare_blockscale, _run_blockscale), "mxfp4": (_prepare_mxfp4, _run_mxfp4),
          "ptgq": (_prepare_ptgq, _run_ptgq), "moe_fp8": (_prepare_moe_fp8, _run_moe_fp8), "moe_mxfp4": (_prepare_moe_mxfp4, _run_moe_mxfp4)}


def prepare(case, seed):
    make, run_ = _KINDS[case["kind"]]
    return run_, case, make(case, _gen(seed))


def run(state):
    run_, case, tensors = state
    return run_(case, tensors)


def work(case):
    kind, N, K = case["kind"], case["N"], case["K"]
    B = case.get("batch", 1)
    w_elem = {"mxfp4": 0.5 + 1 / 32, "moe_mxfp4": 0.5 + 1 / 32}.get(kind, 1.0)          # bytes per weight, scale factors included
    q_elem = 0.0 if kind == "ptgq" else w_elem                                           # the quantized activations are an output too
    if kind.startswith("moe"):
        tokens, rows = case["tokens"], case["tokens"] * case["top_k"]
        weights = min(case["experts"], rows) * N * K
    else:
        tokens = rows = B * case["M"]
        weights = B * N * K
    nbytes = tokens * K * (2 + q_elem) + weights * w_elem + rows * N * 2
    if case.get("mul_add"):
        nbytes += rows * N * 4
    return {"bytes": nbytes, "flops": 2.0 * rows * N * K}


def tolerance(case):
    """Against products of the same operands taken in 64 bits and rounded once to bf16, this path is off by up to 7e-5 (2-norm) and
    by one bf16 step (7.8e-3 of a value) where a sum lies next to a rounding boundary; the bounds are four times that.  The codes
    and scales that the quantizers return are exact, except behind an RMSNorm, whose sum of squares may be taken in any order: a
    code next to a rounding boundary may then land one step (1/16 of a value) away."""
    if case.get("rms"):
        return {"rel": 4e-3, "max": 6e-2, "differ": 1e-3}
    return {"rel": 3e-4, "max": 3.2e-2}


# ---- the same results in 64 bits ---------------------------------------------------------------------

def _e4m3(x, scale):
    """x (fp32) in units of scale, rounded to e4m3: the rule of the FP8 quantizers, whose quotient is the IEEE fp32 one."""
    return (x / scale).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).float()


def _fp8_scale(amax):
    return (amax / torch.full_like(amax, 448.0)).clamp(min=1e-10)


def _exact_rows(x):
    x = x.float()
    scale = _fp8_scale(x.abs().amax(1, keepdim=True))
    return _e4m3(x, scale).double() * scale.double(), scale


def _exact_1x128(x, norm=None):
    x = x.double()
    if norm is not None:
        x = x * (x.square().mean(1, keepdim=True) + EPS).rsqrt() * norm.double()
    g = x.float().view(x.shape[0], -1, 128)
    scale = _fp8_scale(g.abs().amax(2, keepdim=True))
    return (_e4m3(g, scale).double() * scale.double()).view_as(x), scale.squeeze(2)


def _exact_128x128(w):
    N, K = w.shape
    t = w.float().view(N // 128, 128, K // 128, 128)
    scale = _fp8_scale(t.abs().amax((1, 3), keepdim=True))
    return (_e4m3(t, scale).double() * scale.double()).view(N, K)


def _exact_mxfp4(x):
    """Nearest e2m1 magnitude in units of 2^(floor(log2 amax) - 2) per 32 values; a tie goes to the smaller one."""
    g = x.double().view(x.shape[0], -1, 32)
    amax = g.abs().amax(2, keepdim=True)
    e = torch.where(amax > 0, torch.frexp(amax).exponent - 3, -127).clamp(-127, 127)
    unit = torch.ldexp(torch.ones_like(amax), e)
    magnitudes = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64, device=DEV)
    middles = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], dtype=torch.float64, device=DEV)
    q = g / unit
    return (magnitudes[torch.bucketize(q.abs(), middles)] * q.sign() * unit).view(x.shape)


def _exact_pts(c, g):
    B, M, N, K = c["batch"], c["M"], c["N"], c["K"]
    x, xs = _exact_rows(_activations(g, B * M, K))
    w, _ = _exact_rows(_weights(g, B * N, K))
    y = x.view(B, M, K) @ w.view(B, N, K).mT
    if c["bias"]:
        y += torch.randn(B, N, generator=g, device=DEV).bfloat16().double()[:, None]
    return (y[0] if B == 1 else y), None, xs


def _exact_blockscale(c, g):
    M, N, K = c["M"], c["N"], c["K"]
    x = _activations(g, M, K)
    w = _exact_128x128(_weights(g, N, K))
    norm = (1.0 + 0.1 * torch.randn(K, generator=g, device=DEV)).bfloat16() if c["rms"] else None
    x, xs = _exact_1x128(x, norm)
    y = x @ w.T
    if c["mul_add"]:
        c_a, c_b = torch.randn(2, M, N, generator=g, device=DEV).bfloat16().unbind(0)
        y = y * c_a + c_b
    return y, None, xs


def _exact_mxfp4_layer(c, g):
    M, N, K = c["M"], c["N"], c["K"]
    x = _exact_mxfp4(_activations(g, M, K))
    y = x @ _exact_mxfp4(_weights(g, N, K)).T
    if c["mul_add"]:
        c_a, c_b = torch.randn(2, M, N, generator=g, device=DEV).bfloat16().unbind(0)
        y = y * c_a + c_b
    return y, None, None


def _exact_ptgq(c, g):
    B, M, N, K = c["batch"], c["M"], c["N"], c["K"]
    w = _weights(g, B * N, K)
    x = _activations(g, B * M, K).float().view(B, M, K // 64, 64)
    ws = (w.abs().max().float() / 448.0).reshape(1)
    w = _e4m3(w.float(), ws).double().view(B, N, K) * ws.double()
    scale = x.abs().amax(3, keepdim=True).clamp(min=1e-10) * (1.0 / 448.0)
    x = (x * scale.reciprocal()).to(torch.float8_e4m3fn).float().double() * scale.double()
    y = x.view(B, M, K) @ w.mT
    if c["bias"]:
        y += torch.randn(B, 1, N, generator=g, device=DEV).bfloat16().double()
    return y


def _exact_moe_fp8(c, g):
    T, E, N, K, k = c["tokens"], c["experts"], c["N"], c["K"], c["top_k"]
    _, order, hist = _routing(g, T, E, k)
    x, xs = _exact_1x128(_activations(g, T, K))
    y = _empty(T * k, N, dtype=torch.float64)
    at = 0
    for n in hist:
        w = _exact_128x128(_weights(g, N, K))
        torch.matmul(x[order[at: at + n].long() // k], w.T, out=y[at: at + n])
        at += n
    if c["bias"]:
        y += torch.randn(E, N, generator=g, device=DEV).double().repeat_interleave(torch.tensor(hist, device=DEV), 0)
    return y, None, xs


def _exact_moe_mxfp4(c, g):
    T, E, N, K, k = c["tokens"], c["experts"], c["N"], c["K"], c["top_k"]
    _, order, hist = _routing(g, T, E, k)
    x = _exact_mxfp4(_activations(g, T, K))
    gate = torch.rand(T * k, generator=g, device=DEV).double()
    y = _empty(T * k, N, dtype=torch.float64)
    at = 0
    for n in hist:
        w = _exact_mxfp4(_weights(g, N, K))
        ids = order[at: at + n].long()
        y[ids] = (x[ids // k] @ w.T) * gate[ids, None]
        at += n
    return y, None, None


_EXACT = {"pts": _exact_pts, "blockscale": _exact_blockscale, "mxfp4": _exact_mxfp4_layer, "ptgq": _exact_ptgq, "moe_fp8": _exact_moe_fp8,
          "moe_mxfp4": _exact_moe_mxfp4}


def exact(case, seed):
    """What `run` returns, as plain torch gives it: the operands that the rules of the quantizers define, their products in 64 bits.
    None in the place of codes, and for a case of over 1e14 operations."""
    if work(case)["flops"] > 1e14:
        return None
    return _EXACT[case["kind"]](case, _gen(seed))
