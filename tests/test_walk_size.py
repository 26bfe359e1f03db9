"""Shared memory of the weighted walk (ssu_walk_size.hpp): a tree that the form
accepts never asks for more than the kernel's limit, however its nodes fall
into sparse and dense ones; what does not fit is refused (and takes the
embedding).  A host program built from the header checks the arithmetic."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "unifrac-binaries_b200", "csrc")

PROBE = r"""
#include <cstdio>
#include "ssu_walk_size.hpp"
using namespace ssu::walk;
int main() {
    // columns of value-only, sparse and dense rows, each section from a multiple of 32
    auto cols = [](uint32_t value_only, uint32_t sparse, uint32_t dense) {
        auto up = [](uint32_t x) { return (x + 31) / 32 * 32; };
        const uint32_t n = up(up(up(value_only) + sparse) + dense);
        return n < 32 ? 32u : n;
    };
    for (uint32_t n : {0u, 1u, 31u, 33u, 5000u, 39998u, 100000u, 399999u, 524288u, 600001u, 660000u, 700000u, 740000u, 751000u,
                       780000u, 790000u})
        for (uint32_t heights : {0u, 1u, 20u, 300u, 600u, 723u, 1446u, 1973u, 2000u, 3946u, 4095u})
            for (uint32_t part = 0; part < 4; part++) {
                if (!fits(n, heights)) continue;
                const uint32_t bypassed = part == 1 ? n / 2 : 0, sparse = (n - bypassed) / (part + 1);
                const uint32_t c = cols(bypassed, sparse, n - bypassed - sparse);
                for (uint64_t levels : {uint64_t(0), uint64_t(heights), uint64_t(2) * heights}) {
                    if (shared_bytes(c, levels) > kSharedMost) { std::printf("too much %u %u\n", n, heights); return 1; }
                    if (capacity(c, levels) < kValuesLeast / kPerNode && capacity(c, levels) != c) { std::printf("few values\n"); return 2; }
                }
            }
    if (fits(740000, 2000) || fits(751000, 600) || fits(660000, 3946)) { std::printf("accepted\n"); return 3; }
    if (!fits(740000, 300) || !fits(500000, 4095) || !fits(39998, 60)) { std::printf("refused\n"); return 4; }
    std::printf("ok\n");
    return 0;
}
"""


def test_accepted_trees_fit_the_walks_shared_memory(tmp_path):
    src = tmp_path / "walk.cpp"
    src.write_text(PROBE)
    exe = tmp_path / "walk"
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
