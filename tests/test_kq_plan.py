"""The split plan of kq_batch.cu (csrc/kq_plan.cuh, compiled here for the host) over shapes of every size: what a plan puts into
shared memory fits, the partial sums that a cluster sends fit the ring, the sizes do not wrap at the largest planes; and the rule that gives a call to that kernel or to another."""
import os
import subprocess
import sys

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include "kq_plan.cuh"
using namespace kq;
static unsigned long long checked, refused;
static void fail(const char* what, int f, unsigned nt, unsigned k, unsigned n, unsigned b, const Plan& p) {
    std::printf("%s: format %d NT %u K %u N %u tokens %u: S %u clusters %u rounds %u tiles %u ku %u stages %u smem %zu\n", what, f, nt, k, n, b, p.split, p.clusters, p.rounds, p.round_tiles, p.ku, p.stages, p.smem);
    std::exit(1);
}
template <int F, uint32_t NT>
void check(unsigned k, unsigned n, unsigned b, const uint32_t* cap) {
    Plan p;
    if (!make_plan<F, NT>(p, cap, k, n, b)) { ++refused; return; }
    ++checked;
    using T = Fmts<F>;
    const unsigned long long units = k >> 8, tiles = (n + 15ull) / 16, w = kWarps, d = p.stages, rt = p.round_tiles, ku = p.ku;
    auto up = [](unsigned long long v) { return (v + 15) / 16 * 16; };
    const unsigned long long smem = w * d * T::kStage + b * (ku * 1024 + 64) + up(ku * b * 4) + ku * b * T::kBlocks * 4 + (rt + w) * 16 * NT * 8 * 4 + w * d * 8 + 16;
    if (smem != p.smem || smem > kSmemMax) fail("shared memory", F, NT, k, n, b, p);
    if (p.split > kMaxSplit || p.split > units || cap[p.split] == 0 || ku * p.split < units || d < 2) fail("split", F, NT, k, n, b, p);
    // the kernel gives cluster y the tiles [y tiles / clusters, (y + 1) tiles / clusters), in rounds of rt
    if (p.clusters == 0 || p.clusters > tiles || (tiles + p.clusters - 1) / p.clusters > (unsigned long long)p.rounds * rt) fail("rounds", F, NT, k, n, b, p);
    const unsigned long long rpo = (rt * 16 + p.split - 1) / p.split;
    if (p.split > 1 && p.split * b * rpo * 4 > w * d * T::kStage) fail("partial sums", F, NT, k, n, b, p);
}
template <int F>
void all(unsigned k, unsigned n, unsigned b, const uint32_t* cap) {
    if (b <= 8) check<F, 1>(k, n, b, cap); else check<F, 2>(k, n, b, cap);
}
int main() {
    const uint32_t b200[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15}, part[9] = {0, 16, 8, 0, 4, 0, 0, 0, 1};
    for (unsigned k : {256u, 512u, 1024u, 3328u, 5120u, 12288u, 17408u, 40960u, 262144u, 1u << 20, 0x40000000u})
        for (unsigned n : {1u, 5u, 16u, 17u, 512u, 5003u, 27648u, 262144u, 1u << 24, (1u << 29) + 7u, 0x3fffffffu, 0x40000000u})
            for (unsigned b = 1; b <= 16; ++b)
                for (const uint32_t* cap : {b200, part}) {
                    all<kQ4K>(k, n, b, cap); all<kQ40>(k, n, b, cap); all<kQ5K>(k, n, b, cap); all<kQ6K>(k, n, b, cap); all<kQ80>(k, n, b, cap);
                }
    std::printf("%llu plans, %llu without\n", checked, refused);
    return checked > 5000 ? 0 : 2;
}
"""


def test_plans_fit(tmp_path):
    (tmp_path / "plan.cc").write_text(SRC)
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "paddock_b200", "csrc")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", csrc, "-o", str(tmp_path / "plan"), str(tmp_path / "plan.cc")])
    subprocess.check_call([str(tmp_path / "plan")], timeout=120)


def test_routes_of_small_batches():
    """Both sides of every line of the rule (kquant.cu), asked from the library: 1 kq_batch, 2 the integer kernel, 3 tcgen05, 0 other."""
    import paddock_b200
    lib = paddock_b200.KernelPack.load()._lib
    route = lib.pdk_kquant_gemm_route
    q4_0, q4_k, q5_k, q6_k, iq4_xs = 2, 12, 13, 14, 23
    for dtype in (q4_k, q5_k):
        assert route(9216, 27648, 2, dtype) == 2 and route(9472, 27648, 2, dtype) == 1         # K past the integer kernel's image
        # N (tokens + 8) <= 680 sqrt(4096) = 43520
        assert route(4096, 4352, 2, dtype) == 1 and route(4096, 4960, 2, dtype) == 2
        assert route(4096, 2720, 8, dtype) == 1 and route(4096, 2721, 8, dtype) == 2
        # N (K + 2048) <= 30, 20, 10 million up to 2, 4, 8 tokens
        assert route(1024, 9765, 2, dtype) == 1 and route(1024, 9766, 2, dtype) == 2
        assert route(1024, 6510, 4, dtype) == 1 and route(1024, 6511, 4, dtype) == 2
        assert route(1024, 3255, 8, dtype) == 1 and route(1024, 3256, 8, dtype) == 2
        assert route(5120, 25600, 1, dtype) == 0 and route(5120, 25600, 65, dtype) == 0
        assert route(1 << 30, 1 << 30, 8, dtype) == 1 and route(256, (1 << 32) - 1, 2, dtype) == 2
    assert [route(5120, 25600, m, q4_k) for m in (8, 9, 64)] == [2, 3, 3]
    for dtype in (q4_k, q4_0):      # narrow planes, few of tcgen05's work items: kq_batch; 32 tokens are two of its passes
        assert [route(9728, n, 9, dtype) for n in (1100, 3000, 5000)] == [1, 1, 3]
        assert [route(9728, n, 32, dtype) for n in (520, 2560)] == [3, 3]
        assert [route(5120, n, 16, dtype) for n in (1100, 5000)] == [1, 3]
        # long K: kq_batch has room for the partial sums of one tile only, nine rounds of them
        assert route(14848, 2112, 16, dtype) == 3 and route(14848, 704, 16, dtype) == 1
        # more than 32 tokens: what counts is the first 32, which tcgen05 takes in one launch
        assert [route(9216, 640, m, dtype) for m in (32, 33, 37, 64)] == [3, 3, 3, 3]
    assert [route(5120, 25600, m, q5_k) for m in (8, 9, 64)] == [2, 1, 1]
    assert [route(5120, 25600, m, q4_0) for m in (2, 8, 9, 64)] == [1, 1, 3, 3]
    assert [route(5120, 25600, m, q6_k) for m in (2, 16, 64)] == [1, 1, 1]
    assert route(5120, 25600, 4, iq4_xs) == 0


def test_the_switch_is_not_overruled():
    """PDK_Q4K_TC5_MIN by hand: from that many tokens on every Q4_K plane asks tcgen05 first, narrow ones too; 0 = none does."""
    src = """import paddock_b200
route = paddock_b200.KernelPack.load()._lib.pdk_kquant_gemm_route
print([route(9728, 1100, m, 12) for m in (4, 9, 16)], route(9728, 1100, 9, 2))"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    for value, want in ((None, "[1, 1, 1] 1"), ("9", "[1, 3, 3] 3"), ("4", "[3, 3, 3] 3"), ("0", "[1, 1, 1] 1")):
        env = {k: v for k, v in os.environ.items() if k != "PDK_Q4K_TC5_MIN"} | ({"PDK_Q4K_TC5_MIN": value} if value else {})
        assert subprocess.check_output([sys.executable, "-c", src], cwd=root, env=env, text=True).strip() == want, value
