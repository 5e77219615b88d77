"""The split plan of kq_batch.cu (csrc/kq_plan.cuh, compiled here for the host) over shapes of every size: what a plan puts into
shared memory fits, the partial sums that a cluster sends fit the ring, the sizes do not wrap at the largest planes."""
import os
import subprocess

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
                    all<kQ4K>(k, n, b, cap); all<kQ40>(k, n, b, cap); all<kQ5K>(k, n, b, cap); all<kQ6K>(k, n, b, cap);
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
