"""Which launches a mixture-of-experts block on the tensor-core path is made of, on both sides of the by-pair calls' limits
(no GPU: the executor only records)."""
from types import SimpleNamespace

import pytest

from paddock_b200 import planes as P


class Recorder:
    """Stands for GpuExecutor: every call by its name and arguments."""

    def __init__(self):
        self.calls = []
        self.pack = SimpleNamespace(call=lambda name, *args, stream: self.calls.append((name, args)))


def workspace(k, bm, blocks):
    names = ("idx w sorted_row sorted_slot block_expert pair_pos x4q x4s x4step h4q h4s h4step g_raw u_raw h part").split()
    return SimpleNamespace(bm=bm, n_active=k, tokens=4, max_blocks=blocks, sms=148, **{n: n for n in names})


@pytest.mark.parametrize("bm", [8, 32])
@pytest.mark.parametrize("n_expert,k,by_pair", [(128, 16, True), (128, 17, False), (1500, 4, True), (1501, 4, False), (24, 20, False)])
def test_calls_stay_within_the_limits_of_their_entry_points(monkeypatch, n_expert, k, by_pair, bm):
    monkeypatch.setattr(P, "_stream", lambda: 0)
    rows, ex = 4, Recorder()
    planes = SimpleNamespace(n_expert=n_expert, embd=256, ff=128, gate_bias=None, up_bias=None, down_bias=None,
                             tc5={n: ("sf", "meta") for n in ("gate", "up", "down")},
                             **{n: SimpleNamespace(data="data") for n in ("gate", "up", "down")})
    n = P.moe_mxfp4_experts_tc5(ex, planes, workspace(k, bm, 40), "x", rows)
    names = [c[0] for c in ex.calls]
    assert n == len(names) == 5
    paired = {"pdk_moe_align_pos", "pdk_moe_prep_tokens_f4", "pdk_moe_prep_pairs_f4", "pdk_mxfp4_moe_gate_up_tc5"}
    if by_pair:
        assert set(names) <= paired | {"pdk_mxfp4_moe_gemm_tc5_ahead"} and "pdk_moe_prep_tokens_f4" in names
    else:      # by position throughout: gate|up in one launch leaves rows that only the by-pair preparation finds
        assert names == ["moe_align_bm", "pdk_moe_prep_act_f4", "pdk_mxfp4_moe_gemm_tc5_ahead", "pdk_moe_prep_act_f4",
                         "pdk_mxfp4_moe_gemm_tc5_ahead"]
