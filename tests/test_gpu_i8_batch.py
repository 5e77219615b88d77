"""The integer batch kernel (q4k_batch_i8.cu: Q4_K and Q5_K planes wide enough for it, 2..8 tokens; Q4_K with int8 activations too) at
ragged rows, zero and tiny tokens and every K slice count from its smallest.  Each shape's route is asserted, so that a
change of the rule cannot move these calls to another kernel unseen.

Bounds against the f64 product of the dequantized plane.  f32 activations are 15-bit block floating point per 256 elements: a
rounding error of at most 2^-16 of a block's largest |x|, which for normal activations is about four times the mean |x|, so
|error| <= 4 * 2^-16 sum |w||x| = 6.1e-5 without any cancellation.  int8 activations times their f32 scale are 24-bit numbers of 8 bits
each times a block's scale: the same rounding, the same bound."""
import numpy as np
import pytest
import torch

import oracle
from gpu_util import cond_err, dev, dev_f32
from test_gpu_kq_batch import planes

pytestmark = pytest.mark.gpu
DTYPE = {"q4_k": 12, "q5_k": 13}
SHAPES = [(1024, 13999), (2048, 12345), (5120, 9473)]


def make(pack, name, k, n, batch):
    assert pack._lib.pdk_kquant_gemm_route(k, n, batch, DTYPE[name]) == 2
    return planes(pack, name, k, n, 400 + k + batch)


def check(pack, outs, want, x, k, n, batch):
    torch.cuda.synchronize()
    assert pack.device_error() == 0
    assert torch.equal(outs[0], outs[1])
    y = outs[0].cpu().numpy().reshape(batch, n)
    assert np.isfinite(y).all() and not y[0].any()
    ref, ab = oracle.matmul_f64(want, x, k, n, batch, with_abs=True)
    for t in range(1, batch):
        assert cond_err(y[t:t + 1], ref[t:t + 1], np.maximum(ab[t:t + 1], 1e-30)) < 6.1e-5, t


@pytest.mark.parametrize("name", sorted(DTYPE))
@pytest.mark.parametrize("k,n", SHAPES)
@pytest.mark.parametrize("batch", [2, 3, 5, 8])
def test_f32_activations(pack, name, k, n, batch):
    want, d_data, d_sc, dtype = make(pack, name, k, n, batch)
    x = oracle.fill_normal(batch * k, 410 + batch, 1.0)
    x[:k] = 0.0
    x[k:2 * k] *= 1.0e-12
    outs = []
    for _ in range(2):
        outs.append(torch.full((batch * n,), float("nan"), dtype=torch.float32, device="cuda"))
        pack.call("pdk_kquant_gemm_f32", d_data, d_sc, dev_f32(x), outs[-1], k, n, batch, dtype)
    check(pack, outs, want, x, k, n, batch)


@pytest.mark.parametrize("k,n", SHAPES[:2])
@pytest.mark.parametrize("batch", [2, 5, 8])
@pytest.mark.parametrize("slot", ["kquant_gemm_mma_ks", "kquant_gemm_w4a8_sb"])
def test_int8_activations(pack, k, n, batch, slot):
    want, d_data, d_sc, _ = make(pack, "q4_k", k, n, batch)
    x = oracle.fill_normal(batch * k, 420 + batch, 1.0)
    x[:k] = 0.0
    x[k:2 * k] *= 1.0e-12
    q, s, sums = oracle.quantize_q8_act(x)
    xhat = (q.astype(np.float32).reshape(-1, 32) * s.reshape(-1, 1)).reshape(-1)
    d_part = torch.zeros(8 * n * batch, dtype=torch.float32, device="cuda")
    outs = []
    for _ in range(2):
        outs.append(torch.full((batch * n,), float("nan"), dtype=torch.float32, device="cuda"))
        pack.call(slot, d_data, d_sc, dev(q), dev_f32(s), dev_f32(sums), d_part, outs[-1], k, n, batch, 12)
    check(pack, outs, want, xhat, k, n, batch)
