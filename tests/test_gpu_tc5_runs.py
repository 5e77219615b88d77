"""The runs of q4k_tc5.cu: equal runs of unit pairs that cut tiles anywhere (a tile per SM and more), half tiles of even and odd pair counts, one
pair to a tile, ragged rows.  Up to 16 tokens a CTA requests and dequantizes a ring of three boxes (pairs) before it waits for the
activation rows: runs of fewer boxes, of three, of four and of more, with tiles that change inside the ring and without.
Bound: weights rounded to f16, 1e-4 of sum |w||x| as in test_gpu_gemv.py (a weight's rounding is at most 2^-11 of it and a row's add up
like a random walk: the bound is 5 deviations at K = 512, where half a million results of one call reach 1.2e-4)."""
import numpy as np
import pytest
import torch

import oracle
from gpu_util import cond_err, dev, dev_f32
from test_gpu_gemv import KQ, q4k_planes, raw_kquant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n,batch,name", [(512, 6001, 9, "q4_k"), (512, 19000, 16, "q4_0"), (1024, 2561, 16, "q4_k"), (1024, 19001, 20, "q4_k"),
                                            (1536, 9001, 12, "q4_k"), (1536, 20000, 9, "q4_0"), (2560, 19100, 33, "q4_k"), (3584, 12000, 16, "q4_0"),
                                            (1536, 12000, 16, "q4_k"),      # a tile of three boxes a CTA: the ring
                                            (2048, 12000, 9, "q4_0"),       # of four: one more
                                            (1024, 33001, 12, "q4_k")])     # three or four, two to a tile
def test_runs(pack, k, n, batch, name):
    dtype = 12 if name == "q4_k" else 2
    assert pack._lib.pdk_kquant_gemm_route(k, n, batch, dtype) == 3
    if name == "q4_k":
        raw, data, sc = q4k_planes(pack, oracle.fill_normal(n * k, 700 + k, 0.02), n, k)
        want = oracle.dequant_q4_k(raw)
    else:
        ns = n * k // 256
        raw = raw_kquant(name, ns, 700 + k)
        want = oracle.dequant_kquant(name, raw)
        data = torch.zeros(ns * KQ[name][1], dtype=torch.uint8, device="cuda")
        sc = torch.zeros(ns * 24, dtype=torch.uint8, device="cuda")
        pack.call("kquant_repack", dev(raw), data, sc, ns, dtype)
    x = oracle.fill_normal(batch * k, 701 + batch, 1.0)
    outs = []
    for _ in range(3):
        y = torch.full((batch * n,), float("nan"), dtype=torch.float32, device="cuda")
        pack.call("pdk_kquant_gemm_f32", data, sc, dev_f32(x), y, k, n, batch, dtype)
        torch.cuda.synchronize()
        outs.append(y)
    assert pack.device_error() == 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    ref, ab = oracle.matmul_f64(want, x, k, n, batch, with_abs=True)
    assert cond_err(outs[0].cpu().numpy().reshape(batch, n), ref, np.maximum(ab, 1e-30)) < 1e-4
