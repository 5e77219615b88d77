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
from gpu_util import dev_f32, rel_l2
from test_gpu_moe import nvf4_expert_plane

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,n_expert,k,embd,ff,bm,gated,skew", [
    (150, 8, 2, 256, 192, 8, True, 0.0),      # 45 blocks, runs of three to six groups
    (150, 8, 2, 256, 192, 8, True, 3.0),      # most pairs on two experts: runs of a dozen groups, single ones beside them
    (70, 3, 2, 320, 128, 8, False, 1.0),      # one plane, runs that end on every rest of four
    (500, 8, 2, 256, 128, 32, True, 0.0),     # 39 blocks of 32: four to a run
    (500, 8, 2, 192, 320, 32, True, 2.0),     # runs of one block and of a dozen, rests of one to four groups
    (130, 4, 2, 256, 192, 32, False, 0.5),    # 12 blocks: every warp builds the table
    (37, 2, 1, 256, 128, 32, True, 0.0),      # two runs, each with a rest beside a whole block or less than one
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
