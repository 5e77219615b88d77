"""Q8_0 planes times 2 and more tokens where the ring's plan does not hold: kq_batch.cu on int8 codes raised by 128.

Bound: x = hi + lo in f16 keeps 2^-22 of a super-block's largest |x|, but the offset of 128 takes part in the sums, four times the codes'
mean size: 4 x 2^-22 x (largest over mean |x| of a block, about 3) and f32 sums of that size, below 1e-5 of sum |w||x|."""
import pytest
import torch

import oracle
from gpu_util import cond_err, dev_f32
from test_gpu_gemv import q8_planes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n,batch", [(1024, 5, 2), (1280, 17, 3), (1280, 1003, 4), (2304, 33, 5), (5376, 40, 8), (6144, 19, 9), (9472, 48, 16),
                                       (17152, 33, 12), (17408, 16, 33), (5120, 600, 9), (2048, 16400, 2), (27648, 7, 16)])
def test_edges(pack, k, n, batch):
    raw, data, scale = q8_planes(pack, oracle.fill_normal(n * k, 500 + k + n, 0.02), n, k)
    x = oracle.fill_normal(batch * k, 501 + batch, 1.0)
    x[:k] *= 1.0e4
    bias = oracle.fill_normal(n, 502, 0.1)
    outs = []
    for b in (bias, bias, None):
        y = torch.full((batch * n,), float("nan"), dtype=torch.float32, device="cuda")
        pack.call("q8_0_gemm_repacked", data, scale, None if b is None else dev_f32(b), dev_f32(x), y, k, n, batch)
        torch.cuda.synchronize()
        outs.append(y.cpu().numpy().reshape(batch, n))
    assert pack.device_error() == 0
    assert (outs[0] == outs[1]).all()
    ref, ab = oracle.matmul_f64(oracle.dequant_q8_0(raw), x, k, n, batch, with_abs=True)
    for t in range(batch):
        assert cond_err(outs[2][t:t + 1], ref[t:t + 1], ab[t:t + 1]) < 1e-5, t
        assert cond_err(outs[0][t:t + 1] - bias, ref[t:t + 1], ab[t:t + 1] + abs(bias)) < 1e-5, t
