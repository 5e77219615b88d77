"""What the mixture-of-experts calls refuse by their arguments alone, before anything is launched or read (no GPU; the addresses are
made up and no call here gets as far as using them)."""
import ctypes as C

import pytest

import paddock_b200 as pb
from paddock_b200 import pack as packmod

INVALID = 1                   # cudaErrorInvalidValue
A = 0x7000_0000_0000          # an address aligned to anything


def status(name, *args):
    fn = getattr(C.CDLL(pb.lib_path()), name)
    kinds = packmod._EXTRA_SIGS[name]
    assert len(args) == len(kinds)
    fn.argtypes = [packmod._KIND[k] for k in kinds] + [C.c_void_p]
    fn.restype = C.c_int
    return fn(*args, None)


@pytest.mark.parametrize("name", ["pdk_mxfp4_moe_gemm_tc5", "pdk_mxfp4_moe_gemm_tc5_ahead", "pdk_nvf4_moe_gemm_tc5",
                                  "pdk_nvf4_moe_gemm_tc5_ahead", "pdk_mxfp4_moe_gate_up_tc5", "pdk_nvf4_moe_gate_up_tc5"])
@pytest.mark.parametrize("off", [4, 8, 12])
def test_gemm_refuses_scale_records_that_bulk_copies_cannot_read(name, off):
    """The scale records are fetched with cp.async.bulk, which needs 16-byte addresses."""
    rows = A, A + off, A, A, A                                     # xq, xs, xstep, block_expert, sorted_row
    if "gate_up" in name:
        args = (A, A, A, None) * 2 + (A,) + rows + (256, 128, 4, 8, 4, 1.0, 7.0, 0.0)
    else:
        args = (A, A, A, None, A) + (None,) * 5 + rows + (None, None, 256, 128, 4, 8, 4, 2, 0)
    assert status(name, *args) == INVALID


def test_by_pair_calls_refuse_a_missing_position_table():
    """pdk_moe_align_pos refuses it too; the launches would read or write at address 0."""
    assert status("pdk_moe_align_pos", A, A, A, A, None, 4, 2, 8, 8, 8) == INVALID
    assert status("pdk_moe_route_few", A, None, A, A, A, A, A, None, 8, 2, 4, 8, 8) == INVALID
    assert status("pdk_moe_prep_tokens_f4", A, None, A, A, A, 256, 2, 4, 8, 0) == INVALID
    assert status("pdk_moe_prep_pairs_f4", A, None, None, A, A, A, 256, 8, 8, 0, 0, 1.0, 7.0, 0.0) == INVALID
