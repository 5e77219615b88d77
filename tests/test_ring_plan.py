"""The plans of gemv_ring.cu (csrc/ring_plan.cuh, compiled here for the host) over shapes of every size, with the clusters of a B200 and of a
smaller part: the shared memory of a plan fits and its parts do not overlap, warps and stages are what the instances are built for,
every pair of a row has a warp, the sums of a split have room."""
import os
import subprocess

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include "ring_plan.cuh"
using namespace ring;
static unsigned long long checked, refused, kinds[4];
static void fail(const char* what, const char* f, unsigned k, unsigned n, const RingPlan& p) {
    std::printf("%s: %s K %u N %u: W %u teams %u D %u split %u clusters %u smem %u\n", what, f, k, n, p.W, p.teams, p.D, p.split, p.clusters,
                p.smem_bytes);
    std::exit(1);
}
template <class F>
void check(const char* f, unsigned k, unsigned n, const uint32_t* cap) {
    RingPlan p;
    if (!make_plan<F>(k, n, cap, p)) { ++refused; return; }
    ++checked;
    const unsigned long long all = (k + 511ull) / 512, tiles = (n + 15ull) / 16, w = p.W * (unsigned long long)p.teams;
    const bool many = p.teams > 1 || p.W > kMaxWarps;
    ++kinds[(many ? 1 : 0) + (p.split > 1 ? 2 : 0)];
    if (p.W == 0 || p.teams == 0 || p.teams > kMaxTeams || w > (many ? kManyWarps : kMaxWarps) || (many && !F::kMany)) fail("warps", f, k, n, p);
    if (p.D < 2 || p.D > kMaxDepth) fail("depth", f, k, n, p);
    if (p.split == 0 || p.split > kMaxSplit || p.split > all || cap[p.split] == 0) fail("split", f, k, n, p);
    if (p.clusters == 0 || p.clusters > cap[p.split] || p.clusters > tiles) fail("clusters", f, k, n, p);
    unsigned long long most = 0;
    for (unsigned long long r = 0; r < p.split; ++r) {
        const unsigned long long part = (r + 1) * all / p.split - r * all / p.split;
        if (part == 0) fail("empty part", f, k, n, p);
        if (part > most) most = part;
    }
    if (p.k_part < most * 512 || (p.split == 1 && (k & 511) == 0 && p.k_part != k)) fail("activations", f, k, n, p);
    if (p.invariant ? p.W < most : p.W >= most) fail("invariant", f, k, n, p);
    // an invariant warp loads x at its own pair: inside the row, or clamped (a row of an odd number of units)
    const unsigned long long last = all - most;      // where the last, longest part starts
    if (p.invariant && p.split == 1 && p.W != all) fail("idle warps", f, k, n, p);
    if (p.invariant && (last + p.W) * 512 > all * 512) fail("reads past x", f, k, n, p);
    const unsigned long long per = (tiles + p.clusters - 1) / p.clusters, rpo = (per * 16 + p.split - 1) / p.split;
    const unsigned long long stage_data = 2 * (F::kDataBoxes * 2048ull + 16 * F::kHighBytes), stage_rec = 32ull * F::kRecBytes;
    if (p.off_xmeta < 2ull * p.k_part + 32 || p.off_xmeta % 8) fail("limbs", f, k, n, p);
    if (p.off_red < p.off_xmeta + (unsigned long long)p.k_part / F::kBlock * 8) fail("meta", f, k, n, p);
    if (p.off_recv < p.off_red + kRedBufs * w * 64) fail("partial sums", f, k, n, p);
    if (p.off_bar < p.off_recv + (p.split > 1 ? p.split * rpo * 4 : 0) || p.off_bar % 8) fail("sums of the cluster", f, k, n, p);
    if (p.off_rec < p.off_bar + (w * kMaxDepth + 2ull * kRedBufs * p.teams) * 8 + 4 || p.off_rec % 128) fail("barriers", f, k, n, p);
    if (p.off_data < p.off_rec + w * p.D * stage_rec || p.off_data % 1024) fail("records", f, k, n, p);
    if (p.smem_bytes < p.off_data + w * p.D * stage_data || p.smem_bytes > kSmemMax) fail("stages", f, k, n, p);
}
int main() {
    const uint32_t b200[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15}, part[9] = {0, 16, 8, 0, 4, 0, 0, 0, 1};
    for (unsigned k = 256; k <= 32768; k += 256)
        for (unsigned n : {1u, 5u, 16u, 17u, 512u, 1500u, 3200u, 5003u, 9472u, 14000u, 27648u, 262144u, 1u << 24, (1u << 29) + 7u,
                           0x3fffffffu, 0x40000000u})
            for (const uint32_t* cap : {b200, part}) {
                check<Q4KPlane>("Q4_K", k, n, cap); check<Q40Plane>("Q4_0", k, n, cap); check<Q5KPlane>("Q5_K", k, n, cap);
                check<Q6KPlane>("Q6_K", k, n, cap); check<Q80Plane>("Q8_0", k, n, cap);
            }
    for (unsigned k : {65536u, 262144u, 1u << 20, 0x40000000u, 0xffffff00u})
        for (unsigned n : {1u, 1000u, 0x40000000u}) { check<Q4KPlane>("Q4_K", k, n, b200); check<Q80Plane>("Q8_0", k, n, b200); }
    std::printf("%llu plans (one team %llu, many %llu, split %llu, many and split %llu), %llu without\n", checked, kinds[0], kinds[1], kinds[2],
                kinds[3], refused);
    for (unsigned long long v : kinds) if (v < 100) return 2;
    return 0;
}
"""


def test_plans_fit(tmp_path):
    (tmp_path / "plan.cc").write_text(SRC)
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "paddock_b200", "csrc")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", csrc, "-o", str(tmp_path / "plan"), str(tmp_path / "plan.cc")])
    print(subprocess.check_output([str(tmp_path / "plan")], timeout=120, text=True))
