"""The vectorised Q8_0 / Q4_K repack against the any-alignment kernels (a source one element off a 16-byte boundary) and
the oracle, on every remainder of their chunks, random bytes, guard bytes behind the planes."""
import numpy as np
import pytest
import torch

import oracle
from gpu_util import host

pytestmark = pytest.mark.gpu


def run(pack, name, raw, off, n, data_b, scale_b, *extra):
    src = torch.zeros(raw.size + 64, dtype=torch.uint8, device="cuda")
    src[off:off + raw.size] = torch.from_numpy(raw).cuda()
    data = torch.full((n * data_b + 32,), 0xA5, dtype=torch.uint8, device="cuda")
    scale = torch.full((n * scale_b + 32,), 0xA5, dtype=torch.uint8, device="cuda")
    pack.call(name, src[off:], data, scale, n, *extra)
    torch.cuda.synchronize()
    d, s = host(data, np.uint8), host(scale, np.uint8)
    assert (d[n * data_b:] == 0xA5).all() and (s[n * scale_b:] == 0xA5).all()
    return d[:n * data_b], s[:n * scale_b]


@pytest.mark.parametrize("n", [1, 7, 8, 511, 512, 513, 1031])
def test_q8_0(pack, n):
    raw = np.random.default_rng(n).integers(0, 256, n * 34, dtype=np.uint8)
    data, scale = run(pack, "q8_0_repack", raw, 0, n, 32, 2)
    want_data, want_scale = oracle.repack_q8_0(raw)
    assert np.array_equal(data, want_data.view(np.uint8)) and np.array_equal(scale, want_scale.view(np.uint8))
    slow = run(pack, "q8_0_repack", raw, 2, n, 32, 2)
    assert np.array_equal(data, slow[0]) and np.array_equal(scale, slow[1])


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 400])
def test_q4_k(pack, n):
    raw = np.random.default_rng(n).integers(0, 256, n * 144, dtype=np.uint8)
    data, scale = run(pack, "kquant_repack", raw, 0, n, 128, 24, 12)
    assert np.array_equal(data.reshape(n, 128), raw.reshape(n, 144)[:, 16:])
    slow = run(pack, "kquant_repack", raw, 4, n, 128, 24, 12)
    assert np.array_equal(data, slow[0]) and np.array_equal(scale, slow[1])
