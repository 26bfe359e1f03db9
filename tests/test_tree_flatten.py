"""The flattened tree (SYNC_TREE_TABLE of the reference, src/api.cpp:90-92):
one walk that drops the tips without a table row and collapses single-child
nodes on the way must give the rows, lengths (bit for bit), children, parents
and levels that the sheared and collapsed tree gives.  A host program built
from the tree source compares the two over random trees on the CPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "unifrac-binaries_b200", "csrc")

PROBE = r"""
#include <cstdio>
#include <memory>
#include <random>
#include <string>
#include "ssu_tree.hpp"
using namespace ssu;
static std::mt19937_64 rng(7);
static double unit() { return std::uniform_real_distribution<double>(0.0, 1.0)(rng); }
static void grow(int depth, double chain, std::vector<char> &open) {
    open.push_back(1);
    const double x = unit();
    const int kids = depth == 0 || x < 0.15 ? 0 : x < 0.15 + chain ? 1 : x < 0.85 ? 2 : 5;
    for (int i = 0; i < kids; i++) grow(depth - 1, chain, open);
    open.push_back(0);
}
int main() {
    size_t collapsed = 0, empty = 0;
    for (int trial = 0; trial < 600; trial++) {
        std::vector<char> open;
        grow(trial % 9, 0.4 * (trial % 3), open);
        const size_t n = open.size();
        std::unique_ptr<bool[]> o(new bool[n]);
        std::vector<double> len(n, 0.0);
        std::vector<std::string> names(n);
        std::vector<const char *> p(n);
        for (size_t i = 0; i < n; i++) {
            o[i] = open[i] != 0;
            if (o[i]) len[i] = trial % 5 ? unit() : -0.0;
            if (o[i] && i + 1 < n && !open[i + 1]) names[i] = "t" + std::to_string(i);
        }
        for (size_t i = 0; i < n; i++) p[i] = names[i].c_str();
        const BPTree t = BPTree::from_arrays(o.get(), len.data(), p.data(), static_cast<int>(n), false);
        if (t.malformed) return 1;
        const double keep_rate = trial % 4 == 0 ? 1.0 : unit();
        std::vector<int32_t> tags(n, -1);
        NameSet keep;
        for (uint32_t i = 0; i + 1 < n; i++)
            if (t.leaf(i) && unit() < keep_rate) {
                tags[i] = static_cast<int32_t>(rng() % 1000);
                keep.insert(t.name[i]);
            }
        const BPTree c = t.shear(keep).collapse();
        std::vector<int32_t> ctags(c.size(), -1);
        for (uint32_t i = 0; i + 1 < c.size(); i++)
            if (c.leaf(i)) ctags[i] = tags[std::stoul(std::string(c.name[i]).substr(1))];
        collapsed += c.size() < t.size();
        empty += c.size() == 0;
        for (bool bypass : {false, true}) {
            const FlatTree a = flatten(t, tags, bypass), b = flatten(c, ctags, bypass);
            const uint32_t nodes = c.size() ? c.size() / 2 - 1 : 0;
            if (a.n_nodes != nodes || b.n_nodes != nodes || a.n_embedded != b.n_embedded) return 2;
            if (a.length != b.length || a.leaf_obs != b.leaf_obs || a.leaf_rows != b.leaf_rows) return 3;
            if (a.child_ptr != b.child_ptr || a.child_rows != b.child_rows || a.parent != b.parent) return 4;
            if (a.level_ptr != b.level_ptr || a.level_rows != b.level_rows || a.height != b.height) return 5;
            if (a.postorder_row != b.postorder_row) return 6;
            // against the collapsed tree itself: the k-th close is postorder node k
            std::vector<uint32_t> stack;
            uint32_t k = 0;
            for (uint32_t i = 0; i < c.size(); i++) {
                if (c.open[i]) { stack.push_back(i); continue; }
                const uint32_t at = stack.back();
                stack.pop_back();
                if (stack.empty()) break;
                const uint32_t row = a.postorder_row[k++];
                const bool leaf = c.leaf(at);
                if (a.length[row] != c.length[at] || a.leaf_obs[row] != (leaf ? ctags[at] : -1)) return 7;
                if ((row < a.n_embedded) != !(bypass && leaf)) return 8;
                if ((a.height[row] == 0) != leaf) return 9;
                for (uint32_t q = a.child_ptr[row]; q < a.child_ptr[row + 1]; q++)
                    if (a.parent[a.child_rows[q]] != static_cast<int32_t>(row)) return 10;
            }
            if (k != nodes) return 11;
        }
    }
    std::printf("ok %d\n", collapsed > 100 && empty > 0);
    return 0;
}
"""


def test_one_walk_flattens_as_shear_and_collapse_do(tmp_path):
    src = tmp_path / "flatten.cpp"
    src.write_text(PROBE)
    exe = tmp_path / "flatten"
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, str(src), os.path.join(CSRC, "ssu_tree.cpp"), "-pthread",
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok 1", (out.returncode, out.stdout)
