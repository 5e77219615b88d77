"""The ring GEMV (gemv_ring.cu) over its formats and instances: odd super-block counts (the lanes copy the records, the last pair is
half zeros), one and several teams of warps, rows split over a cluster, row counts from one to more tiles than SMs.  test_plans takes shapes
as they come; test_instances looks for a plan of every instance and asserts it.

Bounds as in test_gpu_gemv.py: 15-bit block floating point activations, exact integer products, f32 folds."""
import pytest
import torch

import oracle
from gpu_util import cond_err, dev, dev_f32, gemv_plan, rel_l2
from test_gpu_gemv import KQ, q4k_planes, q8_planes, raw_kquant

pytestmark = pytest.mark.gpu


def plane(pack, name, k, n, seed):
    """-> (weights f32, launch(x, y, stream)) of one plane."""
    if name == "q8_0":
        raw, data, scale = q8_planes(pack, oracle.fill_normal(n * k, seed, 0.02), n, k)
        return oracle.dequant_q8_0(raw), lambda x, y, st=0: pack.call("q8_0_gemv_repacked", data, scale, None, x, y, k, n, stream=st)
    if name == "q4_k":
        raw, data, sc = q4k_planes(pack, oracle.fill_normal(n * k, seed, 0.02), n, k)
        want, dtype = oracle.dequant_q4_k(raw), 12
    else:
        dtype, datab = KQ[name]
        ns = n * k // 256
        raw = raw_kquant(name, ns, seed)
        want = oracle.dequant_kquant(name, raw)
        data = torch.zeros(ns * datab, dtype=torch.uint8, device="cuda")
        sc = torch.zeros(ns * 24, dtype=torch.uint8, device="cuda")
        pack.call("kquant_repack", dev(raw), data, sc, ns, dtype)
    return want, lambda x, y, st=0: pack.call("kquant_gemv", data, sc, x, y, k, n, dtype, stream=st)


DTYPE = {"q8_0": 8, "q4_k": 12, "q4_0": KQ["q4_0"][0], "q5_k": KQ["q5_k"][0], "q6_k": KQ["q6_k"][0]}


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("name", ["q8_0", "q4_k", "q4_0", "q5_k", "q6_k"])
def test_instances(pack, name, many, odd, split):
    """Every instance of the kernel - many warps or one team, odd rows, a cluster per row - at the smallest plane of a list that
    takes it here (clusters of a size that fit the chip differ between parts)."""
    if many and name == "q8_0":
        pytest.skip("no instance: two boxes a unit leave no room for the stages")
    for k, n in sorted(((k, n) for k in range(1536 + 256 * odd, 17408, 512) for n in (523, 1053, 2501, 3203, 4003)), key=lambda s: s[0] * s[1]):
        warps, teams, ctas, _ = gemv_plan(pack, k, n, DTYPE[name])
        if warps != 0 and (teams > 1 or warps > 12) == many and (ctas > 1) == split:
            # the large elements fill whole blocks: in a block with both kinds 15 bits of the largest element alone cost up to 1.2e-5
            # of sum |w||x| at K = 1536 (the f64 product with x rounded to limbs: 1.21e-5 for Q5_K 1536 x 523)
            check(pack, name, k, n, 192)
            return
    pytest.fail("no shape takes this instance")


@pytest.mark.parametrize("name", ["q8_0", "q4_k", "q4_0", "q5_k", "q6_k"])
@pytest.mark.parametrize("k,n", [(1024, 17), (1536, 1), (1792, 333), (2304, 520), (2560, 2501), (3328, 4749), (5376, 17), (9472, 40),
                                 (17152, 531), (17408, 1040), (27904, 5)])
def test_plans(pack, name, k, n):
    check(pack, name, k, n)


def check(pack, name, k, n, tail=200):
    want, launch = plane(pack, name, k, n, 40 + k + n)
    x = oracle.fill_normal(k, 41 + k, 1.0)
    x[k - tail:] *= 100.0                  # the end of the row counts
    x = oracle.bf16_round(x)               # what 15 bits drop of an f32 value would be the larger error where a few elements rule the sum
    outs = []
    for _ in range(2):
        y = torch.full((n,), float("nan"), dtype=torch.float32, device="cuda")
        launch(dev_f32(x), y)
        torch.cuda.synchronize()
        outs.append(y)
    assert pack.device_error() == 0
    assert torch.equal(outs[0], outs[1])
    ref, ab = oracle.matmul_f64(want, x, k, n, 1, with_abs=True)
    y = outs[0].cpu().numpy()
    assert cond_err(y, ref[0], ab[0]) < 1e-5
    assert rel_l2(y, ref[0]) < 1e-4


@pytest.mark.parametrize("name,k", [("q4_k", 9472), ("q6_k", 8448), ("q5_k", 2304), ("q8_0", 5376)])
def test_overlapping_launches_in_a_graph(pack, name, k):
    """Launches that overlap (dependent launch), each on the last one's output, from a graph: the bits of one call at a time."""
    _, launch = plane(pack, name, k, k, 50 + k)
    bufs = [dev_f32(oracle.fill_normal(k, 51, 1.0))] + [torch.zeros(k, dtype=torch.float32, device="cuda") for _ in range(3)]
    want = []
    for i in range(3):
        launch(bufs[i], bufs[i + 1])
        torch.cuda.synchronize()
        want.append(bufs[i + 1].clone())
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        g = torch.cuda.CUDAGraph()
        g.capture_begin()
        for i in range(3):
            launch(bufs[i], bufs[i + 1], s.cuda_stream)
        g.capture_end()
        for b in bufs[1:]:
            b.zero_()
        g.replay()
    torch.cuda.synchronize()
    assert pack.device_error() == 0
    for i in range(3):
        assert torch.equal(bufs[i + 1], want[i]), i
