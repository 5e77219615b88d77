"""Bounded barrier waits as the sources write them: a wait that gives up must be given up by the whole warp.  Lanes can disagree (one
sees the phase complete while another sees the abort flag or the end of its time); the code behind a wait holds warp-wide
instructions (tcgen05.ld is .sync.aligned, shuffles and __syncwarp take the full mask), and a warp of which some lanes left early
never gets past one.  The case itself cannot be made on a GPU without hanging it, so this reads the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "paddock_b200", "csrc")
# the probe and the wait's own test have nothing warp-wide behind their single wait
UNVOTED = {"tc5_probe.cu", "fp8_quant.cu"}
VOTES = ("__all_sync(0xffffffffu", "__syncthreads_or(", "__syncwarp();")


def waits(text):
    """(line number, the statement that waits and the one behind it) of every wait outside the wait functions themselves."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"\b(mbar_wait|mbar_wait_park|wait_for|wait_longer)\(", text):
        start = max(text.rfind(c, 0, m.start()) for c in ";{}")
        statement = text[start + 1:m.start()]
        if re.search(r"\b(bool|return)\s+(tc5::)?$|__forceinline__|__noinline__|return[^;]*$", statement):
            continue       # a definition, or one wait function calling another
        end = text.index(";", text.index(";", m.end()) + 1)
        yield text.count("\n", 0, m.start()) + 1, text[start + 1:end + 1]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))), ids=os.path.basename)
def test_a_wait_is_given_up_by_the_whole_warp(path):
    found = list(waits(open(path).read()))
    if os.path.basename(path) in UNVOTED:
        return
    alone = [line for line, code in found if not any(v in code for v in VOTES)]
    assert not alone, f"{os.path.basename(path)}: waits decided by each lane for itself at lines {alone}"


def test_the_waits_are_found():
    count = {os.path.basename(p): len(list(waits(open(p).read()))) for p in glob.glob(os.path.join(CSRC, "*.cu*"))}
    for name, least in (("moe_grouped.cuh", 5), ("q4k_tc5.cu", 8), ("fp8_gemm2.cu", 4), ("nvf4_gemm2.cu", 4), ("splitk_gemm.cu", 4),
                        ("gemv_ring.cu", 6), ("kq_batch.cu", 1), ("q4k_batch_i8.cu", 1)):
        assert count[name] >= least, (name, count)


def test_a_warp_that_gave_up_still_comes_to_the_named_barriers():
    """The NVFP4 pair kernel's eight epilogue warps meet at a named barrier before and after they fill the output box, and bar.sync
    has no limit: a warp whose accumulator never came must come to all meetings that are left before it leaves the loop."""
    text = open(os.path.join(CSRC, "nvf4_gemm2.cu")).read()
    body = text[text.index("epilogue (both CTAs"):text.index("tma_store_wait_all()")]
    assert [body.count(c) for c in ("bar.sync 2, 256;", "break;")] == [3, 1]
    gave_up = body[body.index("if (!ok) {"):body.index("break;")]
    left = re.search(r"for \(uint32_t left = ([^;]*); left; --left\) asm volatile\(\"bar.sync 2, 256;\"", gave_up).group(1)
    left = left.replace("u ", " ").replace("u;", "").replace("1u", "1").replace("/", "//")
    for n_pairs in (1, 3, 74):
        for n_tiles in (1, 2, 74, 75, 300):
            for pair in range(min(n_pairs, n_tiles)):
                tiles = list(range(pair, n_tiles, n_pairs))
                for i, tile in enumerate(tiles):      # gave up in tile i, between its two meetings
                    assert eval(left, {}, {"n_tiles": n_tiles, "tile": tile, "n_pairs": n_pairs}) == 1 + 2 * (len(tiles) - 1 - i)
