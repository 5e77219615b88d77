"""The runs of q4k_tc5.cu (csrc/q4k_runs.cuh, compiled here for the host): every super-block pair of a plane belongs to one CTA, no tile to
more than two, no CTA is without work."""
import os
import subprocess

SRC = r"""
#include <cstdio>
#include <initializer_list>
#include "q4k_runs.cuh"
using namespace q4k_runs;
int main() {
    unsigned long long seen[3] = {0, 0, 0};
    for (uint32_t sms : {1u, 16u, 132u, 148u})
        for (uint32_t ppt = 1; ppt <= 32u; ++ppt)
            for (uint32_t tiles = 1; tiles <= 700u; ++tiles) {
                const Runs r = pick(tiles, ppt, sms, tiles & 1u ? 16u : 32u);
                bool ok = r.grid >= 1u && r.grid <= sms && start(r, 0u, ppt) == 0u && start(r, r.grid, ppt) == tiles * ppt;
                uint32_t of[700] = {0};
                for (uint32_t c = 0; c < r.grid && ok; ++c) {
                    const uint32_t lo = start(r, c, ppt), hi = start(r, c + 1u, ppt);
                    ok = lo < hi;
                    for (uint32_t t = lo / ppt; ok && t * ppt < hi; ++t) ok = ++of[t] <= 2u;
                }
                if (!ok) {
                    std::printf("tiles %u pairs %u SMs %u: cut %u grid %u base %u extra %u\n", tiles, ppt, sms, r.cut, r.grid, r.base, r.extra);
                    return 1;
                }
                ++seen[r.cut];
            }
    std::printf("%llu %llu %llu\n", seen[0], seen[1], seen[2]);
    return seen[0] > 1000 && seen[1] > 1000 && seen[2] > 1000 ? 0 : 2;
}
"""


def test_runs_cover_the_plane(tmp_path):
    (tmp_path / "runs.cc").write_text(SRC)
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "paddock_b200", "csrc")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", csrc, "-o", str(tmp_path / "runs"), str(tmp_path / "runs.cc")])
    subprocess.check_call([str(tmp_path / "runs")], timeout=120)
