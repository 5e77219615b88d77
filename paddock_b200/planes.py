"""Device planes and operator calls, named after the reference's operator API
(crates/paddock-engine/src/gpu: types.rs plane structs, upload.rs / kquant.rs /
q8_gemm.rs wrappers).  Buffers are torch tensors (torch is the allocator and
stream owner here, as cudarc is for the reference); every compute call goes
through the C ABI of libpaddock_b200.so on the current torch stream.
"""
from dataclasses import dataclass

import torch

from .pack import KernelPack

GGML_Q8_0 = 8
GGML_Q4_K = 12


def _stream():
    """Raw handle of the current stream.  torch.cuda.current_stream() builds a Stream object per call: 3.2 us
    on a B200 host against 0.2 us here, next to 2.4 us for a launch."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


@dataclass
class RepackedQ8:
    """types.rs:482-487: int8 data [out][in] + f16 scale [out][in/32]; dims = (in, out)."""
    data: torch.Tensor
    scale: torch.Tensor
    dims: tuple


@dataclass
class RepackedKQ:
    """types.rs:268-281: k-quant data + 24-byte scale records; dims = (in, out)."""
    data: torch.Tensor
    scales: torch.Tensor
    dims: tuple
    ty: int


class GpuExecutor:
    """The subset of crates/paddock-engine/src/gpu/mod.rs:143-252 that drives the
    quantized linear layer.  Method names and argument meaning follow the Rust
    wrappers; a NULL slot raises MissingOp, a refused launch raises LaunchError."""

    def __init__(self, pack=None, device=None):
        if not torch.cuda.is_available():
            raise RuntimeError("paddock_b200 needs a CUDA device: there is no CPU path")
        torch.cuda.init()
        self.pack = pack or KernelPack.load()
        self.device = torch.device("cuda", torch.cuda.current_device() if device is None else device)

    # -- upload / repack (gpu/upload.rs:305-353, gpu/kquant.rs:284-374) --------
    def upload_raw(self, host_bytes):
        """Raw GGUF tensor bytes (a pinned or pageable uint8 tensor) -> device."""
        return host_bytes.to(self.device, non_blocking=True)

    def repack_q8_blocks(self, raw_dev, in_dim, out_dim):
        n_blocks = in_dim * out_dim // 32
        data = torch.empty(n_blocks * 32, dtype=torch.int8, device=self.device)
        scale = torch.empty(n_blocks, dtype=torch.float16, device=self.device)
        self.pack.call("q8_0_repack", raw_dev, data, scale, n_blocks, stream=_stream())
        return RepackedQ8(data, scale, (in_dim, out_dim))

    def repack_kquant_raw(self, raw_dev, in_dim, out_dim, ty=GGML_Q4_K):
        n_super = in_dim * out_dim // 256
        data = torch.empty(n_super * 128, dtype=torch.uint8, device=self.device)
        scales = torch.empty(n_super * 24, dtype=torch.uint8, device=self.device)
        self.pack.call("kquant_repack", raw_dev, data, scales, n_super, ty, stream=_stream())
        return RepackedKQ(data, scales, (in_dim, out_dim), ty)

    # -- linear calls (gpu/q8_gemm.rs:11-47, gpu/kquant.rs:499-528) --------------
    def q8_0_gemv_repacked(self, w, bias, x, y):
        self.pack.call("q8_0_gemv_repacked", w.data, w.scale, bias, x, y, w.dims[0], w.dims[1], stream=_stream())

    def q8_0_gemm_repacked(self, w, bias, x, y, batch):
        self.pack.call("q8_0_gemm_repacked", w.data, w.scale, bias, x, y, w.dims[0], w.dims[1], batch,
                       stream=_stream())

    def kquant_gemv(self, w, x, y):
        self.pack.call("kquant_gemv", w.data, w.scales, x, y, w.dims[0], w.dims[1], w.ty, stream=_stream())

    def kquant_gemm_f32(self, w, x, y, batch):
        self.pack.call("pdk_kquant_gemm_f32", w.data, w.scales, x, y, w.dims[0], w.dims[1], batch, w.ty,
                       stream=_stream())


@dataclass
class RepackedMxfp4:
    """types.rs:111-127: 16-byte nibble blocks + 1-byte E8M0 scales."""
    data: torch.Tensor
    scale: torch.Tensor


@dataclass
class MoeMxfp4Planes:
    """One MoE layer's expert planes (gate / up: [expert][ff][embd], down: [expert][embd][ff])
    and optional f32 biases ([expert][ff] / [expert][embd])."""
    gate: RepackedMxfp4
    up: RepackedMxfp4
    down: RepackedMxfp4
    n_expert: int
    embd: int
    ff: int
    gate_bias: torch.Tensor = None
    up_bias: torch.Tensor = None
    down_bias: torch.Tensor = None
    tc5: dict = None  # per plane name: (tiled UE4M3 scale records, meta) from prepare_tc5()


def prepare_tc5(ex, planes):
    """Load-time step of the tensor-core expert path: tile each plane's E8M0 scales into UE4M3
    scale records (pdk_mxfp4_tc5_tile_scales).  Costs 1/8 of the scale plane's bytes again."""
    if planes.tc5 is not None:
        return planes
    out = {}
    for name, rows, k in (("gate", planes.ff, planes.embd), ("up", planes.ff, planes.embd),
                          ("down", planes.embd, planes.ff)):
        n_bytes = planes.n_expert * ((rows + 127) // 128) * ((k + 255) // 256) * 2048
        tiled = torch.empty(n_bytes, dtype=torch.uint8, device=ex.device)
        meta = torch.zeros(2, dtype=torch.int32, device=ex.device)
        ex.pack.call("pdk_mxfp4_tc5_tile_scales", getattr(planes, name).scale, tiled, meta, rows, k, planes.n_expert,
                     stream=_stream())
        out[name] = (tiled, meta)
    planes.tc5 = out
    return planes


def repack_mxfp4(ex, raw_dev):
    """gpu/moe_mxfp4.rs:908-936: raw 17-byte blocks -> data + scale planes."""
    n_blocks = raw_dev.numel() // 17
    data = torch.empty(n_blocks * 16, dtype=torch.uint8, device=ex.device)
    scale = torch.empty(n_blocks, dtype=torch.uint8, device=ex.device)
    ex.pack.call("mxfp4_repack", raw_dev, data, scale, n_blocks, stream=_stream())
    return RepackedMxfp4(data, scale)


def _unit_in_gemm(ws, max_blocks, ff, n_expert):
    """Whether the gate|up GEMM applies the gated unit itself.  It then keeps both accumulators in one CTA and writes one plane
    instead of two, but no tile's epilogue runs under the next tile's MMAs.  With 32-token blocks that pays where a CTA has ten
    tiles or more: 1024 tokens, 4 of 128 experts, 2880 x 2880 (40 tiles each) 0.91 of the raw planes' time, 64 experts of 2432 x 1408, 913
    tokens (22) 0.91; 32 experts of 1920 x 896, 130 tokens (3) 1.11, 64 of 1024 x 960, 1547 tokens (6) 1.17; the line
    loses 0.2 % over 70 shapes, 3 % at worst (always the unit 2.7 and 17 %).  With 8-token blocks the raw planes stay in L2 (60
    tokens: 172 against 174 us; 128 tokens on 32 experts of 1024 x 768: 20 against 23), but where tiles of one plane would just need
    a second round over the SMs (one token of 4 experts of 2880 x 2880: 31.9 us a block against 30.3)."""
    tiles = max_blocks * ((ff + 127) // 128)
    return _by_pair(ws, n_expert) and (tiles >= 10 * ws.sms if ws.bm == 32 else tiles <= ws.sms < 2 * tiles)


class MoeWorkspace:
    """Buffers of one MoE block call, sized for `tokens` tokens (allocated once, reused)."""

    def __init__(self, ex, planes, tokens, n_active, bm):
        dev, f32, u32 = ex.device, torch.float32, torch.int32
        pairs = tokens * n_active
        self.bm, self.tokens, self.n_active = bm, tokens, n_active
        self.max_blocks = min(pairs, pairs // bm + planes.n_expert)
        self.sms = torch.cuda.get_device_properties(dev).multi_processor_count if torch.device(dev).type == "cuda" else 148
        nb = self.max_blocks * bm
        self.idx = torch.empty(pairs, dtype=u32, device=dev)
        self.w = torch.empty(pairs, dtype=f32, device=dev)
        self.sorted_row = torch.empty(nb, dtype=u32, device=dev)
        self.sorted_slot = torch.empty(nb, dtype=u32, device=dev)
        self.block_expert = torch.empty(self.max_blocks, dtype=u32, device=dev)
        self.pair_pos = torch.empty(pairs, dtype=u32, device=dev)      # where each (token, slot) pair went
        self.xq = torch.empty(tokens * planes.embd * 2, dtype=torch.uint8, device=dev)
        self.xscale = torch.empty(tokens, dtype=f32, device=dev)
        self.h = torch.zeros(nb * planes.ff, dtype=f32, device=dev)
        self.hq = torch.empty(nb * planes.ff * 2, dtype=torch.uint8, device=dev)
        self.hscale = torch.empty(nb, dtype=f32, device=dev)
        self.part = torch.empty(pairs * planes.embd, dtype=f32, device=dev)
        # tensor-core path: four NVFP4 term rows per block position, raw gate / up outputs
        self.x4q = torch.empty(nb * 4 * planes.embd // 2, dtype=torch.uint8, device=dev)
        self.x4s = torch.zeros(self.max_blocks * ((planes.embd + 255) // 256) * 2048, dtype=torch.uint8, device=dev)
        self.x4step = torch.empty(nb, dtype=f32, device=dev)
        self.h4q = torch.empty(nb * 4 * planes.ff // 2, dtype=torch.uint8, device=dev)
        self.h4s = torch.zeros(self.max_blocks * ((planes.ff + 255) // 256) * 2048, dtype=torch.uint8, device=dev)
        self.h4step = torch.empty(nb, dtype=f32, device=dev)
        self.g_raw = torch.empty(nb * planes.ff, dtype=f32, device=dev)
        self.u_raw = torch.empty(nb * planes.ff, dtype=f32, device=dev)


def moe_mxfp4_experts(ex, planes, ws, x, rows, alpha=1.702, limit=7.0):
    """align -> activation step -> gate|up + SwiGLU -> activation step -> down for `rows` token rows whose
    expert choices and routing weights are already in ws.idx / ws.w ([rows][ws.n_active]); leaves the
    weighted per-(row, slot) outputs in ws.part.  Five launches."""
    st = _stream()
    c = ex.pack.call
    k, bm = ws.n_active, ws.bm
    max_blocks = min(ws.max_blocks, min(rows * k, rows * k // bm + planes.n_expert))
    c("moe_align_bm", ws.idx, ws.sorted_row, ws.sorted_slot, ws.block_expert, rows, k, planes.n_expert, bm,
      max_blocks, stream=st)
    c("pdk_moe_prep_act", x, ws.xq, ws.xscale, planes.embd, rows, stream=st)
    c("pdk_mxfp4_moe_gate_up", planes.gate.data, planes.gate.scale, planes.gate_bias, planes.up.data,
      planes.up.scale, planes.up_bias, ws.sorted_row, ws.block_expert, ws.xq, ws.xscale, ws.h, planes.embd,
      planes.ff, bm, max_blocks, alpha, limit, stream=st)
    c("pdk_moe_prep_act", ws.h, ws.hq, ws.hscale, planes.ff, max_blocks * bm, stream=st)
    c("pdk_mxfp4_moe_down", planes.down.data, planes.down.scale, planes.down_bias, ws.sorted_row, ws.sorted_slot,
      ws.block_expert, ws.w, ws.hq, ws.hscale, ws.part, planes.ff, planes.embd, k, bm, max_blocks, stream=st)
    return 5


def _by_pair(ws, n_expert):
    """Whether the preparations go by (token, slot) pair: pdk_moe_align_pos, which knows the pairs' positions, takes up to 1500
    experts, pdk_moe_prep_tokens_f4 up to 16 pairs of a token.  Other blocks go by position, through calls without these limits."""
    return n_expert <= 1500 and ws.n_active <= 16


def _route_and_prepare(ex, ws, x, rows, embd, n_expert, max_blocks, natural, logits=None, router_bias=None):
    """Positions and term rows of x: top-k (with logits; else ws.idx / ws.w hold the choices already), alignment, one preparation
    per token.  Returns the number of launches."""
    st = _stream()
    c = ex.pack.call
    k, bm = ws.n_active, ws.bm
    tokens = x, ws.pair_pos, ws.x4q, ws.x4s, ws.x4step, embd, k, rows, bm, int(natural)
    if logits is not None and rows <= 8 and rows * k <= 32 and n_expert <= 512 and max_blocks <= 32:
        # decode widths: top-k and alignment in one launch
        c("pdk_moe_route_few", logits, router_bias, ws.idx, ws.w, ws.sorted_row, ws.sorted_slot, ws.block_expert, ws.pair_pos,
          n_expert, k, rows, bm, max_blocks, stream=st)
        c("pdk_moe_prep_tokens_f4", *tokens, stream=st)
        return 2
    n = 2
    if logits is not None:
        c("moe_topk_batch", logits, router_bias, n_expert, k, ws.idx, ws.w, rows, stream=st)
        n = 3
    if not _by_pair(ws, n_expert):
        c("moe_align_bm", ws.idx, ws.sorted_row, ws.sorted_slot, ws.block_expert, rows, k, n_expert, bm, max_blocks, stream=st)
        args = x, None, ws.sorted_row, ws.block_expert, ws.x4q, ws.x4s, ws.x4step, embd, bm, max_blocks, 0, 1.0, 0.0
        c(*(("pdk_moe_prep_act_f4n", *args, 0.0) if natural else ("pdk_moe_prep_act_f4", *args)), stream=st)
        return n
    c("pdk_moe_align_pos", ws.idx, ws.sorted_row, ws.sorted_slot, ws.block_expert, ws.pair_pos, rows, k, n_expert, bm, max_blocks,
      stream=st)
    c("pdk_moe_prep_tokens_f4", *tokens, stream=st)
    return n


def _prepare_unit(ex, ws, x, up, rows, ff, n_expert, max_blocks, mode, natural, alpha, limit, up_add):
    """Term rows for down from what gate|up left: mode 0 the unit's own rows, 1 raw gate and up rows, 2 relu(x)^2."""
    st = _stream()
    if _by_pair(ws, n_expert):
        ex.pack.call("pdk_moe_prep_pairs_f4", x, up, ws.pair_pos, ws.h4q, ws.h4s, ws.h4step, ff, ws.bm, rows * ws.n_active, mode,
                     int(natural), alpha, limit, up_add, stream=st)
        return
    args = x, up, ws.sorted_row, ws.block_expert, ws.h4q, ws.h4s, ws.h4step, ff, ws.bm, max_blocks, mode, alpha, limit
    ex.pack.call(*(("pdk_moe_prep_act_f4n", *args, up_add) if natural else ("pdk_moe_prep_act_f4", *args)), stream=st)


def moe_mxfp4_experts_tc5(ex, planes, ws, x, rows, alpha=1.702, limit=7.0, route=None):
    """moe_mxfp4_experts on the block-scaled tensor-core path (planes prepared with prepare_tc5):
    align -> term rows of x -> gate and up GEMM -> SwiGLU + term rows of h -> down GEMM scattered
    into ws.part.  Returns the number of launches: five, and one more (none at decode widths) with route = (router_logits,
    router_bias), which has the experts chosen here too."""
    st = _stream()
    c = ex.pack.call
    k, bm, t = ws.n_active, ws.bm, planes.tc5
    max_blocks = min(ws.max_blocks, min(rows * k, rows * k // bm + planes.n_expert))
    n = _route_and_prepare(ex, ws, x, rows, planes.embd, planes.n_expert, max_blocks, False, *(route or ()))
    if not _unit_in_gemm(ws, max_blocks, planes.ff, planes.n_expert):
        c("pdk_mxfp4_moe_gemm_tc5_ahead", planes.gate.data, t["gate"][0], t["gate"][1], planes.gate_bias, ws.g_raw,
          planes.up.data, t["up"][0], t["up"][1], planes.up_bias, ws.u_raw, ws.x4q, ws.x4s, ws.x4step,
          ws.block_expert, ws.sorted_row, None, None, planes.embd, planes.ff, planes.n_expert, bm, max_blocks, k, 0,
          stream=st)
        x2, up2, mode = ws.g_raw, ws.u_raw, 1
    else:
        c("pdk_mxfp4_moe_gate_up_tc5", planes.gate.data, t["gate"][0], t["gate"][1], planes.gate_bias,
          planes.up.data, t["up"][0], t["up"][1], planes.up_bias, ws.h, ws.x4q, ws.x4s, ws.x4step, ws.block_expert,
          ws.sorted_row, planes.embd, planes.ff, planes.n_expert, bm, max_blocks, alpha, limit, 1.0, stream=st)
        x2, up2, mode = ws.h, None, 0
    _prepare_unit(ex, ws, x2, up2, rows, planes.ff, planes.n_expert, max_blocks, mode, False, alpha, limit, 1.0)
    c("pdk_mxfp4_moe_gemm_tc5_ahead", planes.down.data, t["down"][0], t["down"][1], planes.down_bias, ws.part,
      None, None, None, None, None, ws.h4q, ws.h4s, ws.h4step, ws.block_expert, ws.sorted_row, ws.sorted_slot,
      ws.w, planes.ff, planes.embd, planes.n_expert, bm, max_blocks, k, 1, stream=st)
    return n + 3


def moe_mxfp4_forward(ex, planes, ws, x, router_logits, out, alpha=1.702, limit=7.0, router_bias=None):
    """The MoE block the way crates/paddock-engine/src/gpu_model/gpt_oss.rs:2279-2521 walks it:
    top-k -> align -> activation step -> gate|up + SwiGLU -> activation step -> down -> combine.
    x f32[tokens][embd], router_logits f32[tokens][n_expert], out f32[tokens][embd] (accumulated into)."""
    st = _stream()
    c = ex.pack.call
    T, k = ws.tokens, ws.n_active
    if planes.tc5 is not None:
        n = moe_mxfp4_experts_tc5(ex, planes, ws, x, T, alpha, limit, route=(router_logits, router_bias))
        c("moe_slot_combine", ws.part, out, planes.embd, k, T, stream=st)
        return n + 1  # launches
    c("moe_topk_batch", router_logits, router_bias, planes.n_expert, k, ws.idx, ws.w, T, stream=st)
    moe_mxfp4_experts(ex, planes, ws, x, T, alpha, limit)
    c("moe_slot_combine", ws.part, out, planes.embd, k, T, stream=st)
    return 7


# ---- NVFP4 expert planes (gpu/types.rs:176-226, Row order) on the same grouped GEMM

@dataclass
class Nvf4MoePlane:
    data: torch.Tensor      # u8 [n_expert*rows][in_dim/2]
    scale: torch.Tensor     # e4m3 [n_expert*rows][in_dim/16]
    scale2: torch.Tensor    # f32 [n_expert]
    n_expert: int
    rows: int
    in_dim: int
    tiled: torch.Tensor = None


def nvf4_moe_prepare(ex, plane):
    """Load-time: tile the plane's per-16 scales into scale records (pdk_nvf4_moe_tile_scales)."""
    if plane.tiled is None:
        n = plane.n_expert * ((plane.rows + 127) // 128) * ((plane.in_dim + 255) // 256) * 2048
        plane.tiled = torch.empty(n, dtype=torch.uint8, device=ex.device)
        ex.pack.call("pdk_nvf4_moe_tile_scales", plane.scale, plane.tiled, plane.rows, plane.in_dim, plane.n_expert,
                     stream=_stream())
    return plane


def moe_nvf4_forward(ex, gate, up, down, ws, x, router_logits, out, gated=True, alpha=1.0, limit=float("inf"),
                     up_add=0.0, router_bias=None):
    """NVFP4 MoE block: top-k -> align -> term rows -> up (and gate) GEMM -> activation + term rows -> down
    GEMM -> combine.  gated: silu-gated unit (plain SwiGLU by default); else relu(up x)^2 (gate ignored).
    ws is a MoeWorkspace built for an object with n_expert / embd / ff attributes."""
    st = _stream()
    c = ex.pack.call
    T, k, bm = ws.tokens, ws.n_active, ws.bm
    n_expert, embd, ff = up.n_expert, up.in_dim, up.rows
    max_blocks = min(ws.max_blocks, min(T * k, T * k // bm + n_expert))
    n = _route_and_prepare(ex, ws, x, T, embd, n_expert, max_blocks, True, router_logits, router_bias)
    if gated and _unit_in_gemm(ws, max_blocks, ff, n_expert):
        c("pdk_nvf4_moe_gate_up_tc5", gate.data, gate.tiled, gate.scale2, None, up.data, up.tiled, up.scale2, None, ws.h,
          ws.x4q, ws.x4s, ws.x4step, ws.block_expert, ws.sorted_row, embd, ff, n_expert, bm, max_blocks, alpha, limit, up_add,
          stream=st)
        x2, up2, mode = ws.h, None, 0
    elif gated:
        c("pdk_nvf4_moe_gemm_tc5_ahead", gate.data, gate.tiled, gate.scale2, None, ws.g_raw, up.data, up.tiled, up.scale2, None,
          ws.u_raw, ws.x4q, ws.x4s, ws.x4step, ws.block_expert, ws.sorted_row, None, None, embd, ff, n_expert, bm,
          max_blocks, k, 0, stream=st)
        x2, up2, mode = ws.g_raw, ws.u_raw, 1
    else:
        c("pdk_nvf4_moe_gemm_tc5_ahead", up.data, up.tiled, up.scale2, None, ws.u_raw, None, None, None, None, None, ws.x4q,
          ws.x4s, ws.x4step, ws.block_expert, ws.sorted_row, None, None, embd, ff, n_expert, bm, max_blocks, k, 0,
          stream=st)
        x2, up2, mode = ws.u_raw, None, 2
    _prepare_unit(ex, ws, x2, up2, T, ff, n_expert, max_blocks, mode, True, alpha, limit, up_add)
    c("pdk_nvf4_moe_gemm_tc5_ahead", down.data, down.tiled, down.scale2, None, ws.part, None, None, None, None, None, ws.h4q,
      ws.h4s, ws.h4step, ws.block_expert, ws.sorted_row, ws.sorted_slot, ws.w, ff, embd, n_expert, bm, max_blocks, k, 1,
      stream=st)
    c("moe_slot_combine", ws.part, out, embd, k, T, stream=st)
    return n + 4  # launches
