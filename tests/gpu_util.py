"""Helpers shared by the -m gpu parity tests: seeded synthetic planes, device
buffers (torch is only the allocator here) and the two error metrics the
reference's own GPU tests use."""
import ctypes

import numpy as np
import torch

import oracle

TOL = 1e-2  # the largest relative error a GEMV / GEMM output may have; the kernels are held to tighter bounds


def dev(a):
    """numpy array -> device tensor with the same bytes."""
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.uint8).reshape(-1)).cuda()


def dev_f32(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def host(t, dtype):
    return t.cpu().numpy().view(dtype)


def seed_for(config, tensor_id):
    return 0x5EED0000 + 256 * config + tensor_id


def bf16_activations(n, seed):
    """N(0,1) rounded to bf16 and widened back to f32 (exact)."""
    return oracle.bf16_round(oracle.fill_normal(n, seed, 1.0))


def cond_err(y, ref, abs_sum):
    """max_i |y - ref| / sum_k |w x|  (tests/gpu_nvfp4_oracle.rs:140-153)."""
    return float(np.max(np.abs(y.astype(np.float64) - ref) / np.maximum(abs_sum, 1e-30)))


def rel_l2(y, ref):
    """rel-L2 (tests/gpu_kquant_parity.rs:145-153)."""
    return float(np.linalg.norm(y.astype(np.float64) - ref) / max(np.linalg.norm(ref), 1e-12))


def gemv_plan(pack, k, n, dtype):
    """(warps of a team, teams, CTAs of a cluster, stages) of the ring kernel for a one-token call; all 0: the register kernel."""
    plan = (ctypes.c_uint32 * 4)()
    assert pack._lib.pdk_gemv_plan(k, n, dtype, plan) == 0
    return tuple(plan)


def gemm_route(pack, k, n, batch, dtype):
    """1 kq_batch.cu, 2 the integer kernel, 3 tcgen05 (K a multiple of 512 up to 16384), 0 none of them."""
    return pack._lib.pdk_kquant_gemm_route(k, n, batch, dtype)
