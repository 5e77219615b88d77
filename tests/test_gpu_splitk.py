"""The K-split FP8 / NVFP4 GEMM at the edges of its plan: one token, whole and ragged token tiles (32, 64, 128, several
of 128), one channel to a ragged last 128-row tile, one K step, and splits that do not divide K (f64 matmul of the
decoded operands; the bounds are those of test_gpu_fp8.py and test_gpu_nvf4.py: exact products, f32 sums)."""
import numpy as np
import pytest
import torch

from gpu_util import cond_err, dev, dev_f32, rel_l2
from test_gpu_fp8 import fp8_case
from test_gpu_nvf4 import check_nvf4_gemm_w4a4

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 256), (1, 127, 2304), (31, 129, 1280), (32, 128, 5120), (33, 640, 256), (64, 1003, 1792), (65, 260, 768),
          (128, 256, 4096), (129, 384, 2560), (385, 136, 1536), (7, 20000, 512),
          # whole tiles to y (short K, or tiles enough) beside meeting partial sums, ragged in tokens and channels
          (33, 1001, 1024), (100, 2500, 512), (257, 1000, 768), (8, 17001, 2048), (6, 130, 17408), (120, 1024, 8192)]


@pytest.mark.parametrize("m,n,k", SHAPES + [(3, 64, 16), (5, 72, 2064)])
@pytest.mark.parametrize("out", ["f32", "bf16"])
def test_fp8(pack, m, n, k, out):
    wq, ws, xq, xs, ref, ab = fp8_case(m, n, k, 900 + m + n)
    d_y = torch.full((m * n,), float("nan"), dtype=torch.float32 if out == "f32" else torch.bfloat16, device="cuda")
    args = dev(wq), dev_f32(ws), dev(xq), dev_f32(xs), d_y, k, n, m
    name = "f8row_gemm" if out == "f32" else "pdk_f8row_gemm_bf16"
    pack.call(name, *args)
    torch.cuda.synchronize()
    first = d_y.clone()
    d_y.fill_(float("nan"))
    pack.call(name, *args)
    torch.cuda.synchronize()
    assert pack.device_error() == 0
    assert torch.equal(first.view(torch.uint8), d_y.view(torch.uint8))      # the partial sums meet in rank order
    y = d_y.float().cpu().numpy().reshape(m, n)
    assert np.isfinite(y).all()
    if out == "f32":
        assert cond_err(y, ref, ab) < 1e-5 and rel_l2(y, ref) < 1e-5
    else:
        assert rel_l2(y, ref) < 4e-3


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("out", ["f32", "bf16"])
def test_nvfp4(pack, m, n, k, out):
    check_nvf4_gemm_w4a4(pack, m, n, k, out)


def test_nvfp4_first_call_behind_its_load(pack):
    """Scale tiler, quantizer and GEMM on fresh buffers with nothing between them: the GEMM requests weights and scale
    records ahead of its wait, behind a quantizer that releases it early, so the tiler makes its stores visible before its
    blocks leave.  Against the same calls with a synchronisation behind each; same bytes."""
    k, n, m = 2048, 640, 5
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(m * k, device="cuda", generator=g)

    def run(w, s, sync):
        tiled = torch.full((((n + 127) // 128) * (k // 256) * 2048,), 0x7F, dtype=torch.uint8, device="cuda")
        xq = torch.zeros(m * k // 2, dtype=torch.uint8, device="cuda")
        xs = torch.zeros(m * k // 16, dtype=torch.uint8, device="cuda")
        y = torch.full((m * n,), float("nan"), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        for call in (("nvf4_tc5_tile_scales", s, tiled, k, n), ("quantize_nvf4", x, xq, xs, m * k),
                     ("nvf4_gemm_tc5w", w, tiled, None, xq, xs, y, 1.0, k, n, m, None, 0)):
            pack.call(*call)
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return y

    for _ in range(20):
        w = torch.randint(0, 256, (n * k // 2,), dtype=torch.uint8, device="cuda", generator=g)
        s = torch.randint(0x28, 0x40, (n * k // 16,), dtype=torch.uint8, device="cuda", generator=g)
        want, got = run(w, s, True), run(w, s, False)
        assert torch.isfinite(want).all() and torch.equal(want, got)
    assert pack.device_error() == 0


def test_fp8_more_channels_than_a_grid_axis_has_tiles(pack):
    """65,536 tiles of 128 channels and one more: tiles are numbered along the grid's first axis, which holds them."""
    k, n = 16, 65536 * 128 + 5
    g = torch.Generator(device="cuda").manual_seed(6)
    w = torch.randint(0, 0x60, (n, k), dtype=torch.uint8, device="cuda", generator=g)
    x = torch.randint(0, 0x60, (1, k), dtype=torch.uint8, device="cuda", generator=g)
    one = torch.ones(n, device="cuda")
    y = torch.full((1, n), float("nan"), device="cuda")
    pack.call("f8row_gemm", w, one, x, one, y, k, n, 1)
    torch.cuda.synchronize()
    assert pack.device_error() == 0
    ref = x.view(torch.float8_e4m3fn).double() @ w.view(torch.float8_e4m3fn).double().t()
    assert float(((y.double() - ref).abs() / ref.clamp_min(1e-30)).max()) < 1e-6      # sixteen exact non-negative products


# The line between tiles of 64 and of 128 tokens, one shape on each side of each of its conditions (296 tiles, 80 tokens on a split
# row, 512 tokens; slabs against tokens and, FP8, long rows of many tiles: below), and second tiles of one and of all but one token.
TILES_64_128 = [(65, 260, 768), (127, 260, 768), (80, 130, 8192), (81, 130, 8192), (129, 300, 5120), (193, 136, 2560), (100, 18944, 256),
                (100, 18945, 256), (512, 136, 768), (513, 136, 768), (90, 5000, 4096), (120, 5000, 4096)]


# (81, 9500, 2816): a CTA of a 64-token tile has 22 slabs, of a 128-token tile 8, and 3 x 14 + 40 is more than 81 tokens but not than 82
@pytest.mark.parametrize("m,n,k", TILES_64_128 + [(81, 9500, 2816), (82, 9500, 2816), (128, 2700, 16640), (129, 2700, 16640)])
def test_fp8_token_tiles(pack, m, n, k):
    test_fp8(pack, m, n, k, "f32")


@pytest.mark.parametrize("m,n,k", TILES_64_128 + [(81, 9500, 5632), (82, 9500, 5632)])
def test_nvfp4_token_tiles(pack, m, n, k):
    check_nvf4_gemm_w4a4(pack, m, n, k, "bf16")
