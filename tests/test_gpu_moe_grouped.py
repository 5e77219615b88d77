"""The grouped expert GEMM where tiles span several blocks of one expert: runs of many 8-token blocks (tiles of four groups with
every rest), runs of 32-token blocks whose rest joins the tile in front or takes one of its own, more than 32 blocks (the table
built by one warp) and fewer (by every warp), one and two planes.

Error: each activation keeps four NVFP4 terms, the group's remainder below 1e-3 of its largest element; the block's result stays
within 2e-3 (2-norm) of the f64 layer, the bound of the other MoE tests."""
import numpy as np
import pytest
import torch

import oracle
from paddock_b200 import planes as P
from gpu_util import dev, dev_f32, rel_l2
from test_gpu_moe import make_layer, nvf4_expert_plane

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,n_expert,k,embd,ff,bm,gated,skew", [
    (150, 8, 2, 256, 192, 8, True, 0.0),      # 45 blocks, runs of three to six groups
    (150, 8, 2, 256, 192, 8, True, 3.0),      # most pairs on two experts: runs of a dozen groups, single ones beside them
    (70, 3, 2, 320, 128, 8, False, 1.0),      # one plane, runs that end on every rest of four
    (500, 8, 2, 256, 128, 32, True, 0.0),     # 39 blocks of 32: four to a run
    (500, 8, 2, 192, 320, 32, True, 2.0),     # runs of one block and of a dozen, rests of one to four groups
    (130, 4, 2, 256, 192, 32, False, 0.5),    # 12 blocks: every warp builds the table
    (37, 2, 1, 256, 128, 32, True, 0.0),      # two runs, each with a rest beside a whole block or less than one
    (3000, 5, 2, 128, 64, 8, True, 0.7),      # 755 blocks: runs that span many of a warp's 32 blocks
    (2600, 40, 3, 64, 64, 8, False, 0.0),     # 1015 blocks
    (6000, 7, 4, 64, 128, 32, False, 0.5),    # 757 blocks of 32
    (300, 16, 4, 1600, 1088, 32, True, 1.0),  # long K: the ring turns inside a tile, tiles alternate between accumulators
    (200, 4, 2, 2112, 640, 8, True, 1.0),     # the same with runs of a dozen groups of 8
])
def test_tiles_over_runs_of_blocks(pack, tokens, n_expert, k, embd, ff, bm, gated, skew):
    ex = P.GpuExecutor(pack)
    gate, wg = nvf4_expert_plane(ex, n_expert, ff, embd, 1000)
    up, wu = nvf4_expert_plane(ex, n_expert, ff, embd, 2000)
    down, wd = nvf4_expert_plane(ex, n_expert, embd, ff, 3000)
    x = oracle.bf16_round(oracle.fill_normal(tokens * embd, 4000, 1.0)).reshape(tokens, embd)
    logits = oracle.fill_normal(tokens * n_expert, 4001, 1.0).reshape(tokens, n_expert)
    logits = (logits - skew * np.arange(n_expert, dtype=np.float32)).astype(np.float32).reshape(-1)

    class Shape:
        pass
    shape = Shape()
    shape.n_expert, shape.embd, shape.ff = n_expert, embd, ff
    ws = P.MoeWorkspace(ex, shape, tokens, k, bm)
    out = torch.zeros(tokens * embd, dtype=torch.float32, device="cuda")
    P.moe_nvf4_forward(ex, gate, up, down, ws, dev_f32(x.reshape(-1)), dev_f32(logits), out, gated=gated)
    torch.cuda.synchronize()
    assert pack.device_error() == 0
    idx, w = oracle.moe_topk(logits, n_expert, k)
    idx, w = idx.reshape(tokens, k), w.reshape(tokens, k)
    ref = np.zeros((tokens, embd))
    for e in range(n_expert):
        t, s = np.nonzero(idx == e)
        xe = x[t].astype(np.float64)
        u = xe @ wu[e].T
        g = xe @ wg[e].T
        h = g / (1.0 + np.exp(-g)) * u if gated else np.maximum(u, 0.0) ** 2
        np.add.at(ref, t, w[t, s][:, None] * (h @ wd[e].T))
    y = out.cpu().numpy().reshape(tokens, embd)
    assert np.isfinite(y).all()
    assert rel_l2(y, ref) < 2e-3
    # every row by itself: a tile that took another expert's weights, or missed a group, is a whole row wrong
    rows = np.linalg.norm(y - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert rows.max() < 1e-2


@pytest.mark.parametrize("tokens,n_expert,k,embd,bm,skew", [
    (9, 8, 2, 128, 8, 0.0),
    (64, 128, 4, 512, 8, 0.0),
    (128, 5, 4, 288, 8, 2.0),         # half a warp in the last slab; runs of a dozen blocks
    (300, 16, 4, 4352, 32, 1.0),      # a row of more groups than threads
    (700, 128, 8, 256, 32, 0.0),      # 5600 pairs: more chunks per warp than it holds in registers
    (1, 512, 16, 64, 8, 0.0),
    (8, 128, 4, 2880, 8, 0.0),        # the widest pdk_moe_route_few takes
    (8, 2, 2, 256, 8, 0.0),
    (2, 512, 8, 256, 32, 0.0),
    (3000, 64, 1, 64, 32, 4.0),       # one token of 64 per expert at best, a thousand blocks; positions staged in shared memory
    (9000, 16, 8, 32, 8, 0.0),        # too many positions for that: written where they go
])
@pytest.mark.parametrize("natural", [False, True])
def test_positions_and_token_rows_equal_the_gathered_ones(pack, tokens, n_expert, k, embd, bm, skew, natural):
    """pdk_moe_align_pos leaves moe_align_bm's tables and, per pair, its position;
    pdk_moe_prep_tokens_f4 then writes, byte for byte, the rows that pdk_moe_prep_act_f4(n) gathers for these positions."""
    c = P.GpuExecutor(pack).pack.call
    pairs = tokens * k
    max_blocks = min(pairs, pairs // bm + n_expert)
    nb = max_blocks * bm
    x = dev_f32(oracle.bf16_round(oracle.fill_normal(tokens * embd, 7, 1.0)))
    logits = oracle.fill_normal(tokens * n_expert, 8, 1.0).reshape(tokens, n_expert)
    logits = dev_f32((logits - skew * np.arange(n_expert, dtype=np.float32)).reshape(-1))
    i32, u8 = torch.int32, torch.uint8
    new = lambda n, dt: torch.zeros(n, dtype=dt, device="cuda")
    t = [dict(idx=new(pairs, i32), w=new(pairs, torch.float32), row=new(nb, i32), slot=new(nb, i32), blk=new(max_blocks, i32),
              q=new(nb * 4 * embd // 2, u8), s=new(max_blocks * ((embd + 255) // 256) * 2048, u8), step=new(nb, torch.float32))
         for _ in range(2)]
    a, b = t
    pos = new(pairs, i32)
    c("moe_topk_batch", logits, None, n_expert, k, a["idx"], a["w"], tokens)
    c("moe_align_bm", a["idx"], a["row"], a["slot"], a["blk"], tokens, k, n_expert, bm, max_blocks)
    args = x, None, a["row"], a["blk"], a["q"], a["s"], a["step"], embd, bm, max_blocks, 0, 1.0, 7.0
    c(*(("pdk_moe_prep_act_f4n", *args, 0.0) if natural else ("pdk_moe_prep_act_f4", *args)))
    b["idx"], b["w"] = a["idx"], a["w"]
    c("pdk_moe_align_pos", b["idx"], b["row"], b["slot"], b["blk"], pos, tokens, k, n_expert, bm, max_blocks)
    if tokens <= 8 and pairs <= 32 and max_blocks <= 32:
        few = {n: torch.full_like(b[n], 3) for n in ("idx", "w", "row", "slot", "blk")}
        few_pos = new(pairs, i32)
        c("pdk_moe_route_few", logits, None, few["idx"], few["w"], few["row"], few["slot"], few["blk"], few_pos, n_expert, k, tokens,
          bm, max_blocks)
        used = (b["blk"] != -1).repeat_interleave(bm)
        for n in few:
            ta, tb = (few[n][used], b[n][used]) if n in ("row", "slot") else (few[n], b[n])
            assert torch.equal(ta.view(u8), tb.view(u8)), n
        assert torch.equal(few_pos, pos)
    c("pdk_moe_prep_tokens_f4", x, pos, b["q"], b["s"], b["step"], embd, k, tokens, bm, int(natural))
    torch.cuda.synchronize()
    assert pack.device_error() == 0
    # unused blocks keep what they had in every table
    for name in a:
        assert torch.equal(a[name].view(u8), b[name].view(u8)), name
    # what the by-pair preparation of position rows leaves, against the call that walks every position; bytes of padding aside
    h, u = (torch.randn(nb * embd, device="cuda", generator=torch.Generator(device="cuda").manual_seed(s)) for s in (5, 6))
    for mode in ((0, 1, 2) if natural else (0, 1)):
        u1 = u if mode == 1 else None
        both = []
        for by_pair in (False, True):
            q, sc, st = torch.zeros_like(a["q"]), torch.zeros_like(a["s"]), torch.zeros_like(a["step"])
            if by_pair:
                c("pdk_moe_prep_pairs_f4", h, u1, pos, q, sc, st, embd, bm, pairs, mode, int(natural), 1.7, 7.0, 1.0)
            elif mode == 0:     # as a gather of each position's own row
                own = torch.where(a["row"] == -1, a["row"], torch.arange(nb, dtype=i32, device="cuda"))
                args = h, None, own, a["blk"], q, sc, st, embd, bm, max_blocks, 0, 1.0, 7.0
                c(*(("pdk_moe_prep_act_f4n", *args, 0.0) if natural else ("pdk_moe_prep_act_f4", *args)))
            else:
                args = h, u1, a["row"], a["blk"], q, sc, st, embd, bm, max_blocks, mode, 1.7, 7.0
                c(*(("pdk_moe_prep_act_f4n", *args, 1.0) if natural else ("pdk_moe_prep_act_f4", *args)))
            both.append((q, sc, st))
        for v, w in zip(*both):
            assert torch.equal(v.view(u8), w.view(u8)), mode
    p = torch.arange(pairs, device="cuda")
    at = (pos.long() & 0x3FFFFFFF)
    assert torch.equal(b["row"][at].long(), p // k) and torch.equal(b["slot"][at].long(), p % k)
    # the positions follow the oracle's grouping: expert of the block a pair landed in, pairs of an expert in order
    idx = torch.from_numpy(oracle.moe_topk(logits.cpu().numpy(), n_expert, k)[0].astype(np.int64)).cuda().view(-1)
    assert torch.equal(b["blk"][at // bm].long(), idx)
    order = torch.argsort(idx * pairs + p)
    assert (at[order][1:] > at[order][:-1]).all()


def test_pairs_without_an_expert_have_no_position(pack):
    c = P.GpuExecutor(pack).pack.call
    idx = torch.tensor([0, -1, 1, 5, 0, 1], dtype=torch.int32, device="cuda")     # two of them outside [0, 2)
    new = lambda n: torch.full((n,), -7, dtype=torch.int32, device="cuda")
    row, slot, blk, pos = new(16), new(16), new(2), new(6)
    c("pdk_moe_align_pos", idx, row, slot, blk, pos, 6, 1, 2, 8, 2)
    torch.cuda.synchronize()
    assert pos.tolist() == [0, -1, 8, -1, 1, 9] and blk.tolist() == [0, 1]
    assert row.tolist() == [0, 4] + [-1] * 6 + [2, 5] + [-1] * 6


@pytest.mark.parametrize("bm", [8, 32])
def test_more_than_sixteen_choices_of_a_token(pack, bm):
    """The caller's own choices may be more than the by-pair preparation takes of a token: the block then goes by position."""
    tokens, n_expert, k, embd, ff = 5, 24, 20, 128, 192
    ex = P.GpuExecutor(pack)
    raw, _ = make_layer(n_expert, embd, ff, 1500, False)
    planes = P.prepare_tc5(ex, P.MoeMxfp4Planes(*(P.repack_mxfp4(ex, dev(raw[n])) for n in ("gate", "up", "down")), n_expert, embd, ff))
    x = oracle.bf16_round(oracle.fill_normal(tokens * embd, 1501, 1.0))
    rng = np.random.default_rng(1502)
    idx = np.stack([rng.permutation(n_expert)[:k] for _ in range(tokens)]).astype(np.uint32)
    w = (rng.random((tokens, k)) / k).astype(np.float32)
    ws = P.MoeWorkspace(ex, planes, tokens, k, bm)
    ws.idx.view(torch.uint8).copy_(dev(idx))
    ws.w.copy_(dev_f32(w).view(-1))
    P.moe_mxfp4_experts_tc5(ex, planes, ws, dev_f32(x), tokens)
    torch.cuda.synchronize()
    assert pack.device_error() == 0
    ref = oracle.moe_mxfp4_layer(raw["gate"], raw["up"], raw["down"], x, idx, w, tokens, k, embd, ff, None, None, None)
    y = ws.part.cpu().numpy().reshape(tokens, k, embd).astype(np.float64).sum(axis=1)
    assert rel_l2(y, ref) < 2e-3


@pytest.mark.parametrize("tokens,n_expert,k,embd,ff,bm,fmt", [
    (1, 64, 4, 512, 384, 8, "mxfp4"),        # up to 32 blocks: every warp builds the tile table; top-k and alignment in one launch
    (8, 16, 4, 256, 192, 8, "nvfp4"),
    (40, 4, 2, 256, 192, 32, "nvfp4"),       # up to 32 blocks of 32
    (60, 32, 4, 320, 256, 8, "mxfp4"),       # more than 32 blocks: one warp builds it
    (300, 16, 4, 256, 320, 32, "nvfp4"),
])
@pytest.mark.parametrize("graph", [False, True])
def test_blocks_of_different_routing_in_a_row(pack, tokens, n_expert, k, embd, ff, bm, fmt, graph):
    """Calls on one workspace with other logits each time and nothing between them give the bits of calls by themselves: the GEMMs
    read the routing tables before their own wait for the kernel in front, on SMs that read the call before's."""
    ex = P.GpuExecutor(pack)
    shape = P.MoeMxfp4Planes(None, None, None, n_expert, embd, ff)
    if fmt == "nvfp4":
        planes = tuple(nvf4_expert_plane(ex, n_expert, r, c, s)[0] for r, c, s in ((ff, embd, 1000), (ff, embd, 2000), (embd, ff, 3000)))
        forward = lambda *a: P.moe_nvf4_forward(ex, *planes, *a)
    else:
        raw, _ = make_layer(n_expert, embd, ff, 1600, False)
        shape = P.prepare_tc5(ex, P.MoeMxfp4Planes(*(P.repack_mxfp4(ex, dev(raw[n])) for n in ("gate", "up", "down")), n_expert, embd, ff))
        forward = lambda *a: P.moe_mxfp4_forward(ex, shape, *a)
    calls = 12
    # skewed one way and the other, so that runs and tiles change from call to call
    tilt = np.linspace(-2.0, 2.0, n_expert, dtype=np.float32)
    logits = [dev_f32(oracle.fill_normal(tokens * n_expert, 1700 + i, 1.0).reshape(tokens, n_expert) + tilt * (i % 3 - 1)).view(-1)
              for i in range(calls)]
    xs = [dev_f32(oracle.bf16_round(oracle.fill_normal(tokens * embd, 1800 + i, 1.0))) for i in range(calls)]
    alone, row = (torch.zeros(calls, tokens * embd, device="cuda") for _ in range(2))
    for i in range(calls):
        forward(P.MoeWorkspace(ex, shape, tokens, k, bm), xs[i], logits[i], alone[i])
        torch.cuda.synchronize()
    ws = P.MoeWorkspace(ex, shape, tokens, k, bm)
    every = lambda: [forward(ws, xs[i], logits[i], row[i]) for i in range(calls)]
    every()
    torch.cuda.synchronize()
    if graph:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            every()
        for _ in range(3):
            row.zero_()
            g.replay()
        torch.cuda.synchronize()
    assert pack.device_error() == 0
    assert bool(alone.any(dim=1).all()) and torch.equal(row, alone)


@pytest.mark.parametrize("rows,k,embd", [
    (1, 1, 4), (5, 3, 1020), (1023, 4, 512),
    (1024, 4, 512), (1024, 5, 516),           # both sides of several rows a block; the last of them has none left over
    (3001, 9, 36), (20001, 2, 4),             # rows of no whole number of warps; a row of four columns
    (2500, 1, 1028), (5000, 2, 640),          # more rows than blocks
    (2400, 4, 260),
])
def test_slot_combine_adds_every_row_once(pack, rows, k, embd):
    """residual += the slots' rows, added up in slot order: bit for bit, and nothing behind the last row."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    part = torch.randn(rows, k, embd, device="cuda", generator=g)
    res = torch.randn(rows + 3, embd, device="cuda", generator=g)
    acc = torch.zeros(rows, embd, device="cuda")
    for s in range(k):
        acc = acc + part[:, s]
    want = res.clone()
    want[:rows] += acc
    pack.call("moe_slot_combine", part, res, embd, k, rows)
    torch.cuda.synchronize()
    assert pack.device_error() == 0 and torch.equal(res, want)


UNITS = {"clamped": (1.702, 7.0, 1.0), "swiglu": (1.0, float("inf"), 0.0), "tight": (1.2, 0.5, 0.25)}   # tight: most values reach the limit


@pytest.mark.parametrize("tokens,n_expert,k,in_dim,out_dim,bm,skew,unit", [
    (1, 8, 4, 320, 384, 8, 0.0, "clamped"),       # tiles of one group, one token in it
    (37, 2, 1, 256, 128, 32, 0.0, "swiglu"),      # a run of one block and a rest
    (150, 8, 2, 448, 320, 8, 3.0, "tight"),       # runs of a dozen groups of 8, a ragged last row tile
    (60, 32, 4, 2112, 136, 8, 0.0, "clamped"),    # long K: the ring turns inside a tile; eight rows in the last row tile
    (300, 16, 4, 1600, 200, 32, 1.0, "swiglu"),   # runs of one to many blocks, tiles of one to six groups
    (700, 64, 2, 256, 256, 32, 0.0, "tight"),     # more than 32 blocks, 22 tokens an expert
    (2000, 24, 2, 576, 256, 32, 0.3, "clamped"),  # several tiles a CTA under its one pair of accumulators
])
@pytest.mark.parametrize("fmt", ["mxfp4", "nvf4"])
def test_gate_and_up_under_one_operand_equal_raw_planes_and_the_unit(pack, tokens, n_expert, k, in_dim, out_dim, bm, skew, unit, fmt):
    """pdk_*_moe_gate_up_tc5 against the unit, in f64, of the raw rows that one-plane calls leave.  Both kernels sum a row in the
    same order, so what may differ is the unit's f32 arithmetic: __expf is within 2 + 1.173 |x| ulp (CUDA's bound), the sigmoid takes
    over at most that, and the sum, the quotient, the two products and the second factor's sum round once each."""
    c = P.GpuExecutor(pack).pack.call
    alpha, limit, up_add = UNITS[unit]
    gen = torch.Generator(device="cuda").manual_seed(tokens + out_dim)
    rand = lambda lo, hi, n: torch.randint(lo, hi, (n,), dtype=torch.uint8, device="cuda", generator=gen)
    norm = lambda *n: torch.randn(*n, device="cuda", generator=gen)
    new = lambda n, dt=torch.int32: torch.zeros(n, dtype=dt, device="cuda")
    pairs, slabs, row_tiles, u8 = tokens * k, (in_dim + 255) // 256, (out_dim + 127) // 128, torch.uint8
    max_blocks = min(pairs, pairs // bm + n_expert)
    nb = max_blocks * bm
    logits = norm(tokens, n_expert) - skew * torch.arange(n_expert, device="cuda")
    idx, w, row, slot, blk = new(pairs), new(pairs, torch.float32), new(nb), new(nb), new(max_blocks)
    c("moe_topk_batch", logits.view(-1), None, n_expert, k, idx, w, tokens)
    c("moe_align_bm", idx, row, slot, blk, tokens, k, n_expert, bm, max_blocks)
    planes = []
    for _ in range(2):
        data, tiled = rand(0, 256, n_expert * out_dim * in_dim // 2), new(n_expert * row_tiles * slabs * 2048, u8)
        if fmt == "mxfp4":
            factor = new(2)
            c("pdk_mxfp4_tc5_tile_scales", rand(117, 122, n_expert * out_dim * in_dim // 32), tiled, factor, out_dim, in_dim, n_expert)
        else:
            factor = (torch.rand(n_expert, device="cuda", generator=gen) + 0.5) * 0.02
            c("pdk_nvf4_moe_tile_scales", rand(0x20, 0x40, n_expert * out_dim * in_dim // 16), tiled, out_dim, in_dim, n_expert)
        planes.append((data, tiled, factor, norm(n_expert * out_dim)))
    x = norm(tokens * in_dim)
    xq, xs, step = new(nb * 4 * in_dim // 2, u8), new(max_blocks * slabs * 2048, u8), new(nb, torch.float32)
    prep_args = x, None, row, blk, xq, xs, step, in_dim, bm, max_blocks, 0, 1.0, 7.0
    prepare = lambda: c(*(("pdk_moe_prep_act_f4", *prep_args) if fmt == "mxfp4" else ("pdk_moe_prep_act_f4n", *prep_args, 0.0)))
    rows = xq, xs, step, blk, row
    dims = in_dim, out_dim, n_expert, bm, max_blocks
    one = (None,) * 5
    gemm = f"pdk_{'mxfp4' if fmt == 'mxfp4' else 'nvf4'}_moe_gemm_tc5"
    raw = [torch.full((nb, out_dim), -7.5, device="cuda") for _ in range(6)]
    part = [torch.zeros(pairs, out_dim, device="cuda") for _ in range(2)]
    prepare()
    for p in range(2):
        c(gemm, *planes[p], raw[p], *one, *rows, None, None, *dims, k, 0)
    c(gemm, *planes[0], part[0], *one, *rows, slot, w, *dims, k, 1)
    # the calls that begin under a preparation in front of them
    prepare()
    c(gemm + "_ahead", *planes[0], raw[2], *planes[1], raw[3], *rows, None, None, *dims, k, 0)
    prepare()
    c(gemm + "_ahead", *planes[0], part[1], *one, *rows, slot, w, *dims, k, 1)
    prepare()
    c(gemm.replace("gemm", "gate_up"), *planes[0], *planes[1], raw[4], *rows, *dims, alpha, limit, up_add)
    torch.cuda.synchronize()
    assert pack.device_error() == 0
    assert torch.equal(raw[0], raw[2]) and torch.equal(raw[1], raw[3]) and torch.equal(part[0], part[1]) and bool(part[0].any())
    used = (blk != -1).repeat_interleave(bm) & (row != -1)
    assert int(used.sum()) == pairs
    assert bool((raw[4][~used] == -7.5).all())                       # rows of padding are left alone
    g, u = raw[0][used].double(), raw[1][used].double()
    xg, yu = g.clamp(max=limit), u.clamp(-limit, limit)
    ref = xg / (1.0 + torch.exp(-alpha * xg)) * (yu + up_add)
    if np.isfinite(limit):
        assert 0.0 < float((g > limit).double().mean()) < 1.0 or unit == "clamped"
    bound = ((2.0 + 1.173 * (alpha * xg).abs() + 6.0) * 2.0 ** -23) * ref.abs() + 1e-30
    assert bool(((raw[4][used].double() - ref).abs() <= bound).all())
