"""kq_batch.cu (Q4_K, Q5_K, Q6_K, Q4_0, up to 16 tokens per launch) at the edges of its plan: one super-block, odd super-block
counts, K too long for one CTA's activations, one row to ragged tiles, one to several rounds per CTA.

Bound: the codes and scales are exact and x = hi + lo in f16 keeps 2^-22 of a super-block's largest |x|, so what is left is that
and the f32 sums: a few 1e-7 of sum |w||x|; 3e-6 leaves room for the blocks whose |w||x| is small beside their largest |x|."""
import numpy as np
import pytest
import torch

import oracle
from gpu_util import cond_err, dev, dev_f32
from test_gpu_gemv import KQ, raw_kquant

pytestmark = pytest.mark.gpu

FORMATS = {**{f: KQ[f] for f in ("q5_k", "q6_k", "q4_0")}, "q4_k": (12, 128)}


def planes(pack, name, k, n, seed):
    dtype, datab = FORMATS[name]
    ns = n * k // 256
    if name == "q4_k":
        raw = oracle.quantize_q4_k(oracle.fill_normal(n * k, seed, 0.02))
        want = oracle.dequant_q4_k(raw)
    else:
        raw = raw_kquant(name, ns, seed)
        want = oracle.dequant_kquant(name, raw)
    d_data = torch.zeros(ns * datab, dtype=torch.uint8, device="cuda")
    d_sc = torch.zeros(ns * 24, dtype=torch.uint8, device="cuda")
    pack.call("kquant_repack", dev(raw), d_data, d_sc, ns, dtype)
    return want, d_data, d_sc, dtype


@pytest.mark.parametrize("name", sorted(FORMATS))
@pytest.mark.parametrize("k,n,batch", [(256, 5, 2), (768, 16, 3), (1280, 17, 8), (5120, 1003, 4), (17408, 40, 7),
                                       (40960, 19, 5), (1280, 33, 9), (2304, 48, 16), (17408, 33, 16), (3328, 130, 33)])
def test_edges(pack, name, k, n, batch):
    want, d_data, d_sc, dtype = planes(pack, name, k, n, 300 + k + n)
    x = oracle.fill_normal(batch * k, 301 + batch, 1.0)
    x[:k] *= 1.0e4
    x[k:2 * k] *= 1.0e-12
    if batch > 2:
        x[2 * k:3 * k] = 0.0
    outs = []
    for _ in range(2):
        d_y = torch.full((batch * n,), float("nan"), dtype=torch.float32, device="cuda")
        pack.call("pdk_kquant_gemm_f32", d_data, d_sc, dev_f32(x), d_y, k, n, batch, dtype)
        torch.cuda.synchronize()
        outs.append(d_y)
    assert pack.device_error() == 0
    assert torch.equal(outs[0], outs[1])
    y = outs[0].cpu().numpy().reshape(batch, n)
    ref, ab = oracle.matmul_f64(want, x, k, n, batch, with_abs=True)
    for t in range(batch):
        assert cond_err(y[t:t + 1], ref[t:t + 1], np.maximum(ab[t:t + 1], 1e-30)) < 3e-6, t
    if batch > 2:
        assert not y[2].any()


@pytest.mark.parametrize("name", sorted(FORMATS))
@pytest.mark.parametrize("batch", [5, 12])
def test_one_token_that_is_not_finite(pack, name, batch):
    """An infinite and a NaN activation reach their own token alone: the other tokens keep their bits."""
    k, n = 1280, 40                       # an odd super-block count: no other kernel takes 12 tokens
    _, d_data, d_sc, dtype = planes(pack, name, k, n, 350)
    x = oracle.fill_normal(batch * k, 351 + batch, 1.0).reshape(batch, k)
    outs = []
    for bad in (False, True):
        if bad:
            x[1, 3], x[3, 700] = np.inf, np.nan
        y = torch.full((batch, n), 7.0, dtype=torch.float32, device="cuda")
        pack.call("pdk_kquant_gemm_f32", d_data, d_sc, dev_f32(x.reshape(-1)), y, k, n, batch, dtype)
        torch.cuda.synchronize()
        outs.append(y)
    assert pack.device_error() == 0
    keep = [t for t in range(batch) if t not in (1, 3)]
    assert torch.equal(outs[0][keep], outs[1][keep]) and torch.isfinite(outs[0]).all()
    assert not torch.isfinite(outs[1][[1, 3]]).any()


@pytest.mark.parametrize("name,batch", [("q6_k", 8), ("q6_k", 12), ("q5_k", 16)])
def test_several_rounds_of_a_cluster(pack, name, batch):
    """5120 x 25600: more partial tiles than shared memory holds at 12 and 16 tokens, so that a ring refills where the
    cluster's partial sums were.  Against an f64 product of the dequantized plane; the same bits every time."""
    k, n = 5120, 25600
    dtype, datab = FORMATS[name]
    ns = n * k // 256
    d_raw = dev(raw_kquant(name, ns, 77))
    d_data = torch.zeros(ns * datab, dtype=torch.uint8, device="cuda")
    d_sc = torch.zeros(ns * 24, dtype=torch.uint8, device="cuda")
    w = torch.zeros(n, k, dtype=torch.float32, device="cuda")
    pack.call("kquant_repack", d_raw, d_data, d_sc, ns, dtype)
    pack.call("kquant_dequant", d_raw, w, ns, dtype)
    x = dev_f32(oracle.fill_normal(batch * k, 78, 1.0)).view(batch, k)
    first = None
    for _ in range(20):
        y = torch.full((batch, n), float("nan"), dtype=torch.float32, device="cuda")
        pack.call("pdk_kquant_gemm_f32", d_data, d_sc, x, y, k, n, batch, dtype)
        first = y if first is None else first
        assert torch.equal(first, y)
    assert pack.device_error() == 0
    for lo in range(0, n, 6400):
        wd = w[lo:lo + 6400].double()
        ref, ab = x.double() @ wd.t(), x.double().abs() @ wd.abs().t()
        assert float(((first[:, lo:lo + 6400].double() - ref).abs() / ab).max()) < 3e-6
