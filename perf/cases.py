"""The work a host program gives this kernel pack, as measurable cases.

Three kinds of call reach the pack:

  linear  y = x . W^T of one quantized weight plane.  Tokens in flight decide what it is: one token is a decode step
          of one sequence, a few to some tens a batched decode or a speculative verify, hundreds to thousands a
          prompt.  GGUF planes (Q8_0 and the k-quants) serve decode and small batches from f32 activations; FP8 and
          NVFP4 planes serve every width and start with the activation quantizer, as the engine's linear call does.
  moe     one mixture-of-experts block: routing, the experts' gated unit, the weighted sum onto the residual.
  load    raw GGUF blocks, already on the device, into the pack's planes: once per tensor when a model is loaded.

Weights and activations are seeded draws of the distributions trained models show (weights N(0, 0.02), activations
N(0, 1) rounded to bf16, router logits N(0, 1)) in the formats' own encodings.
"""
import math

import torch

from paddock_b200 import planes as P
from paddock_b200 import synth
from paddock_b200.planes import GpuExecutor

# GGUF formats of the linear path: ggml type id, bytes and elements of a raw block, bytes of the repacked data plane
# per 256 weights (Q8_0 has its own repack call)
GGUF = {"q8_0": (8, 34, 32, 256), "q4_k": (12, 144, 256, 128), "q5_k": (13, 176, 256, 160),
        "q6_k": (14, 210, 256, 192), "q4_0": (2, 18, 32, 128)}
MAX_ELEMS = 5120 * 27648          # the largest plane of the ranges
MAX_FLOPS = 2 * 4096 * 5120 * 27648


def listed():
    return [
        # the smallest call of a decode step: a key or value projection of a grouped-query attention
        {"name": "q8_0 kv projection, 1 token", "op": "linear", "fmt": "q8_0", "k": 5120, "n": 1024, "m": 1},
        # the wide gate / up projection of a feed-forward layer, one sequence decoding
        {"name": "q4_k gate projection, 1 token", "op": "linear", "fmt": "q4_k", "k": 5120, "n": 25600, "m": 1},
        # the same plane under a batch of sequences
        {"name": "q4_k gate projection, 16 tokens", "op": "linear", "fmt": "q4_k", "k": 5120, "n": 25600, "m": 16},
        # a down projection in the wider k-quant mixed files keep for it; three drafted tokens; a pruned, odd width
        {"name": "q6_k down projection, 3 tokens", "op": "linear", "fmt": "q6_k", "k": 17408, "n": 5003, "m": 3},
        # an attention output projection under a handful of decoding sequences
        {"name": "fp8 output projection, 7 tokens", "op": "linear", "fmt": "fp8", "k": 5120, "n": 5120, "m": 7},
        # a prompt through a gate / up projection
        {"name": "fp8 gate projection, 4096 tokens", "op": "linear", "fmt": "fp8", "k": 5120, "n": 17408, "m": 4096},
        {"name": "nvfp4 gate projection, 1 token", "op": "linear", "fmt": "nvfp4", "k": 5120, "n": 17408, "m": 1},
        # a ragged prompt
        {"name": "nvfp4 gate projection, 1000 tokens", "op": "linear", "fmt": "nvfp4", "k": 5120, "n": 17408, "m": 1000},
        # one sequence, a batch of sequences and a prompt through a block of 128 experts, 4 per token
        {"name": "mxfp4 experts, 1 token", "op": "moe", "fmt": "mxfp4", "e": 128, "a": 4, "k": 2880, "n": 2880, "m": 1},
        {"name": "nvfp4 experts, 60 tokens", "op": "moe", "fmt": "nvfp4", "e": 128, "a": 4, "k": 2880, "n": 2880, "m": 60},
        {"name": "mxfp4 experts, 1024 tokens", "op": "moe", "fmt": "mxfp4", "e": 128, "a": 4, "k": 2880, "n": 2880, "m": 1024},
        {"name": "q4_k load", "op": "load", "fmt": "q4_k", "k": 5120, "n": 25600},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    op = rng.choice(["gguf"] * 5 + ["fp8", "fp8", "nvfp4", "nvfp4", "moe", "moe", "load"])
    if op == "moe":
        return {"op": "moe", "fmt": rng.choice(["mxfp4", "nvfp4"]), "e": rng.choice([32, 64, 128]), "a": rng.choice([2, 4, 8]),
                "k": _log(rng, 1024, 2880, 64), "n": _log(rng, 768, 2880, 64), "m": _log(rng, 1, 512)}
    if op == "load":
        fmt = rng.choice(["q4_k", "q8_0"])
        k = _log(rng, 1024, 17408, 256)
        return {"op": "load", "fmt": fmt, "k": k, "n": _log(rng, 512, min(27648, MAX_ELEMS // k))}
    if op == "gguf":
        fmt = rng.choice(["q8_0", "q4_k", "q4_k", "q5_k", "q6_k", "q4_0"])
        # rows are whole blocks: 256 weights for the k-quants and their 256-weight planes, 32 for Q8_0
        k = _log(rng, 1024, 17408, 64 if fmt == "q8_0" and rng.random() < 0.3 else 256)
        n = _log(rng, 512, min(27648, MAX_ELEMS // k), rng.choice([1, 64, 128]))
        return {"op": "linear", "fmt": fmt, "k": k, "n": n, "m": 1 if rng.random() < 0.5 else _log(rng, 2, 32)}
    k = _log(rng, 1024, 17408, 256)
    n = _log(rng, 512, min(27648, MAX_ELEMS // k), rng.choice([8, 64, 128]))
    m = _log(rng, 1, 8192) if rng.random() < 0.6 else _log(rng, 1, 64)
    return {"op": "linear", "fmt": op, "k": k, "n": n, "m": min(m, MAX_FLOPS // (2 * k * n))}


# ---------------------------------------------------------------- inputs
_EXECUTOR = None


def _executor():
    """One executor per process, as a host program has."""
    global _EXECUTOR
    if _EXECUTOR is None:
        _EXECUTOR = GpuExecutor()
    return _EXECUTOR


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _raw_gguf(fmt, elems, seed):
    """Raw blocks of a tensor.  Q8_0 and Q4_K are quantized from N(0, 0.02); the other formats have no quantizer here
    and take uniform codes under small positive block scales."""
    if fmt == "q8_0":
        return synth.quantize_q8_0(synth.normal(elems, seed, 0.02, "cuda"))
    if fmt == "q4_k":
        return synth.quantize_q4_k(synth.normal(elems, seed, 0.02, "cuda"))
    _, nbytes, per, _ = GGUF[fmt]
    g = torch.Generator(device="cuda").manual_seed(seed)
    raw = torch.randint(0, 256, (elems // per, nbytes), dtype=torch.uint8, device="cuda", generator=g)
    d = (torch.rand(elems // per, device="cuda", generator=g) * 1e-3 + 1e-4).to(torch.float16)
    d = d.view(torch.uint8).view(-1, 2)
    at = 208 if fmt == "q6_k" else 0
    raw[:, at:at + 2] = d
    if fmt == "q5_k":
        raw[:, 2:4] = d.flip(0)
    return raw.reshape(-1)


def _gguf_plane(ex, fmt, k, n, seed):
    raw = _raw_gguf(fmt, n * k, seed)
    if fmt == "q8_0":
        return ex.repack_q8_blocks(raw, k, n)
    if fmt == "q4_k":
        return ex.repack_kquant_raw(raw, k, n)
    ty, _, _, per256 = GGUF[fmt]
    units = n * k // 256
    data = torch.empty(units * per256, dtype=torch.uint8, device="cuda")
    scales = torch.empty(units * 24, dtype=torch.uint8, device="cuda")
    ex.pack.call("kquant_repack", raw, data, scales, units, ty, stream=_stream())
    return P.RepackedKQ(data, scales, (k, n), ty)


_E2M1_CUTS = (0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0)


def _e2m1(v):
    """Code of the nearest e2m1 value, sign in bit 3."""
    cuts = torch.tensor(_E2M1_CUTS, device=v.device)
    return torch.bucketize(v.abs(), cuts).to(torch.uint8) | ((v < 0).to(torch.uint8) << 3)


def _mxfp4_plane(rows, k, n_expert, gen):
    """Expert weights N(0, 0.02): 32-weight blocks, E8M0 scale 2^(floor(log2 amax) - 2), nibble j and j + 16 in byte j."""
    data = torch.empty(n_expert, rows * k // 32, 16, dtype=torch.uint8, device="cuda")
    scale = torch.empty(n_expert, rows * k // 32, dtype=torch.uint8, device="cuda")
    for e in range(n_expert):
        b = torch.randn(rows * k // 32, 32, device="cuda", generator=gen) * 0.02
        s = torch.floor(torch.log2(b.abs().amax(dim=1))) - 2.0
        c = _e2m1(b * torch.exp2(-s)[:, None])
        data[e] = c[:, :16] | (c[:, 16:] << 4)
        scale[e] = (s + 127.0).to(torch.uint8)
    return P.RepackedMxfp4(data.view(-1), scale.view(-1))


def _nvfp4_codes(b):
    """f32 [blocks][16] -> (bytes [blocks][8] with the even element in the low nibble, e4m3 scale bytes [blocks])."""
    s = (b.abs().amax(dim=1) / 6.0).to(torch.float8_e4m3fn)
    c = _e2m1(b / s.float().clamp_min(2.0 ** -9)[:, None])
    return c[:, 0::2] | (c[:, 1::2] << 4), s.view(torch.uint8)


_NVFP4_GAIN = 2048.0   # N(0, 0.02) weights are scaled up into the e4m3 range of the block scales; scale2 undoes it


def _nvfp4_expert_plane(ex, rows, k, n_expert, gen):
    data = torch.empty(n_expert, rows * k // 16, 8, dtype=torch.uint8, device="cuda")
    scale = torch.empty(n_expert, rows * k // 16, dtype=torch.uint8, device="cuda")
    for e in range(n_expert):
        b = torch.randn(rows * k // 16, 16, device="cuda", generator=gen) * (0.02 * _NVFP4_GAIN)
        data[e], scale[e] = _nvfp4_codes(b)
    scale2 = torch.full((n_expert,), 1.0 / _NVFP4_GAIN, device="cuda")
    return P.nvf4_moe_prepare(ex, P.Nvf4MoePlane(data.view(-1), scale.view(-1), scale2, n_expert, rows, k))


def _prepare_moe(ex, case, seed):
    e, a, k, n, m = case["e"], case["a"], case["k"], case["n"], case["m"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["fmt"] == "mxfp4":
        gate, up, down = (_mxfp4_plane(r, c, e, gen) for r, c in ((n, k), (n, k), (k, n)))
        shape = P.prepare_tc5(ex, P.MoeMxfp4Planes(gate, up, down, e, k, n))
        planes = shape
    else:
        planes = tuple(_nvfp4_expert_plane(ex, r, c, e, gen) for r, c in ((n, k), (n, k), (k, n)))
        shape = P.MoeMxfp4Planes(None, None, None, e, k, n)      # the workspace needs the sizes only
    ws = P.MoeWorkspace(ex, shape, m, a, 8 if m * a <= 1024 else 32)
    x = synth.bf16_round(synth.normal(m * k, seed + 1000, 1.0, "cuda"))
    logits = synth.normal(m * e, seed + 2000, 1.0, "cuda")
    residual = synth.normal(m * k, seed + 3000, 1.0, "cuda")
    return {"ex": ex, "case": case, "planes": planes, "ws": ws, "x": x, "logits": logits, "residual": residual}


def _prepare_fp(ex, case, seed):
    """An FP8 or NVFP4 plane, its activations and the buffers of one linear call."""
    k, n, m = case["k"], case["n"], case["m"]
    w = synth.normal(n * k, seed, 0.02, "cuda")
    s = {"ex": ex, "case": case, "x": synth.bf16_round(synth.normal(m * k, seed + 1000, 1.0, "cuda")),
         "y": torch.empty(m, n, dtype=torch.bfloat16, device="cuda")}
    if case["fmt"] == "fp8":
        s["w"] = torch.empty(n * k, dtype=torch.uint8, device="cuda")
        s["w_scale"] = torch.empty(n, dtype=torch.float32, device="cuda")
        ex.pack.call("bf16_to_f8row", w.to(torch.bfloat16), s["w"], s["w_scale"], k, n, stream=_stream())
        s["xq"] = torch.empty(m * k, dtype=torch.uint8, device="cuda")
        s["x_scale"] = torch.empty(m, dtype=torch.float32, device="cuda")
        return s
    data, scale = _nvfp4_codes(w.view(-1, 16) * _NVFP4_GAIN)
    s["w"] = data.view(-1)
    s["w_scale"] = torch.zeros(((n + 127) // 128) * (k // 256) * 2048, dtype=torch.uint8, device="cuda")
    ex.pack.call("nvf4_tc5_tile_scales", scale.view(-1), s["w_scale"], k, n, stream=_stream())
    s["xq"] = torch.empty(m * k // 2, dtype=torch.uint8, device="cuda")
    s["x_scale"] = torch.empty(m * k // 16, dtype=torch.uint8, device="cuda")
    return s


def prepare(case, seed):
    ex = _executor()
    if case["op"] == "moe":
        return _prepare_moe(ex, case, seed)
    if case["op"] == "load":
        return {"ex": ex, "case": case, "raw": _raw_gguf(case["fmt"], case["n"] * case["k"], seed)}
    if case["fmt"] in ("fp8", "nvfp4"):
        return _prepare_fp(ex, case, seed)
    k, n, m = case["k"], case["n"], case["m"]
    return {"ex": ex, "case": case, "plane": _gguf_plane(ex, case["fmt"], k, n, seed),
            "x": synth.bf16_round(synth.normal(m * k, seed + 1000, 1.0, "cuda")),
            "y": torch.empty(m, n, dtype=torch.float32, device="cuda")}


# ---------------------------------------------------------------- the calls
def run(state):
    ex, case = state["ex"], state["case"]
    op, fmt = case["op"], case["fmt"]
    if op == "load":
        plane = (ex.repack_q8_blocks if fmt == "q8_0" else ex.repack_kquant_raw)(state["raw"], case["k"], case["n"])
        return [plane.data, plane.scale if fmt == "q8_0" else plane.scales]
    if op == "moe":
        args = state["ws"], state["x"], state["logits"], state["residual"]
        if fmt == "mxfp4":
            P.moe_mxfp4_forward(ex, state["planes"], *args)
        else:
            P.moe_nvf4_forward(ex, *state["planes"], *args)
        return state["residual"]      # accumulated onto, as a layer does
    k, n, m, x, y = case["k"], case["n"], case["m"], state["x"], state["y"]
    if fmt in ("fp8", "nvfp4"):
        call, stream = ex.pack.call, _stream()
        if fmt == "fp8":
            call("quantize_e4m3_row", x, state["xq"], state["x_scale"], k, m, stream=stream)
            call("pdk_f8row_gemm_bf16", state["w"], state["w_scale"], state["xq"], state["x_scale"], y, k, n, m, stream=stream)
        else:
            call("quantize_nvf4", x, state["xq"], state["x_scale"], m * k, stream=stream)
            call("pdk_nvf4_gemm_bf16", state["w"], state["w_scale"], None, state["xq"], state["x_scale"], y,
                 1.0 / _NVFP4_GAIN, k, n, m, stream=stream)
        return y
    plane = state["plane"]
    if fmt == "q8_0":
        if m == 1:
            ex.q8_0_gemv_repacked(plane, None, x, y)
        else:
            ex.q8_0_gemm_repacked(plane, None, x, y, m)
    elif m == 1:
        ex.kquant_gemv(plane, x, y)
    else:
        ex.kquant_gemm_f32(plane, x, y, m)
    return y


# ---------------------------------------------------------------- what a pass cannot do without
def _weight_bytes(fmt, elems):
    if fmt in GGUF:
        return elems * GGUF[fmt][1] / GGUF[fmt][2]
    return elems * {"fp8": 1.0, "nvfp4": 0.5625, "mxfp4": 0.53125}[fmt]


def work(case):
    op, fmt, k, n = case["op"], case["fmt"], case["k"], case["n"]
    if op == "load":     # raw blocks in, planes out (k-quant scale records are 24 bytes per 256 weights)
        out = n * k / 32 * 34 if fmt == "q8_0" else n * k / 256 * 152
        return {"bytes": _weight_bytes(fmt, n * k) + out, "flops": 0}
    m = case["m"]
    if op == "moe":      # the experts that m tokens reach, x and logits in, the residual in and out
        reached = case["e"] * (1.0 - (1.0 - case["a"] / case["e"]) ** m)
        return {"bytes": reached * _weight_bytes(fmt, 3 * k * n) + m * (12 * k + 4 * case["e"]),
                "flops": 6.0 * m * case["a"] * k * n}
    y = 2 if fmt in ("fp8", "nvfp4") else 4
    return {"bytes": _weight_bytes(fmt, n * k) + 4 * m * k + y * m * n, "flops": 2.0 * m * n * k}


def tolerance(case):
    op, fmt = case["op"], case["fmt"]
    if op == "load":
        return "exact"
    if op == "moe":
        return {"rel": 1e-3, "max": 2e-2}     # activations in four 4-bit terms: 2e-4 of the block's result
    if fmt in ("fp8", "nvfp4"):
        return {"rel": 4e-3, "max": 3e-2}     # bf16 results
    if case["m"] >= 9 and fmt == "q4_k" or case["m"] >= 4 and fmt == "q4_0":
        return {"rel": 1e-3, "max": 1e-2}     # weights rounded to f16 on the tensor cores
    return {"rel": 1e-4, "max": 2e-3}         # 15-bit activations, exact weights, f32 sums
