// Host-side phylogeny handling: BP trees, newick, shear, collapse, flatten.
#include "ssu_tree.hpp"

#include "ssu_host.hpp"

#include <algorithm>
#include <cstdlib>

namespace ssu {

void BPTree::check_parentheses() {
    int64_t depth = 0, least = 0;
    for (uint8_t o : open) {
        depth += o ? 1 : -1;
        least = std::min(least, depth);
    }
    malformed = depth != 0 || least < 0;
}

std::vector<uint32_t> BPTree::partners() const {
    std::vector<uint32_t> match(open.size(), 0), stack(open.size() + 1);
    size_t top = 0;
    for (uint32_t i = 0; i < open.size(); i++) {
        if (open[i]) {
            stack[top++] = i;
        } else if (top > 0) {
            const uint32_t o = stack[--top];
            match[o] = i;
            match[i] = o;
        }
    }
    return match;
}

BPTree BPTree::from_arrays(const bool *structure, const double *lengths, const char *const *names, int n,
                           bool copy_names) {
    BPTree t;
    const uint32_t m = n > 0 ? static_cast<uint32_t>(n) : 0;
    t.open.resize(m);
    t.length.resize(m);
    t.name.resize(m);
    if (copy_names) t.storage = std::make_shared<std::deque<std::string>>();
    for (uint32_t i = 0; i < m; i++) {
        t.open[i] = structure[i] ? 1 : 0;
        t.length[i] = lengths[i];
        const char *nm = names[i] ? names[i] : "";
        if (copy_names) {
            t.storage->emplace_back(nm);
            t.name[i] = t.storage->back();
        } else {
            t.name[i] = nm;
        }
    }
    t.check_parentheses();
    return t;
}

namespace {

// Rooted tree as child lists, the intermediate form of the newick parser.
struct ChildTree {
    std::vector<std::vector<uint32_t>> children;
    std::vector<double> length;
    std::vector<std::string> name;
    uint32_t add() {
        children.emplace_back();
        length.push_back(0.0);
        name.emplace_back();
        return static_cast<uint32_t>(children.size() - 1);
    }
};

BPTree serialise(const ChildTree &ct, uint32_t root) {
    BPTree t;
    t.storage = std::make_shared<std::deque<std::string>>(ct.name.begin(), ct.name.end());
    const std::deque<std::string> &names = *t.storage;
    const size_t n = 2 * ct.children.size();
    t.open.reserve(n);
    t.length.reserve(n);
    t.name.reserve(n);
    // explicit stack: (node, next child index)
    std::vector<std::pair<uint32_t, uint32_t>> stack;
    stack.emplace_back(root, 0);
    t.open.push_back(1);
    t.length.push_back(ct.length[root]);
    t.name.push_back(names[root]);
    while (!stack.empty()) {
        auto &top = stack.back();
        const auto &kids = ct.children[top.first];
        if (top.second < kids.size()) {
            uint32_t c = kids[top.second++];
            t.open.push_back(1);
            t.length.push_back(ct.length[c]);
            t.name.push_back(names[c]);
            stack.emplace_back(c, 0);
        } else {
            t.open.push_back(0);
            t.length.push_back(0.0);
            t.name.emplace_back("");  // a NUL-terminated empty name
            stack.pop_back();
        }
    }
    t.check_parentheses();
    return t;
}

void apply_label(ChildTree &ct, uint32_t node, const std::string &label) {
    if (label.empty()) return;
    const size_t colon = label.find_last_of(':');
    if (colon == std::string::npos) {
        ct.name[node] = label;
        ct.length[node] = 0.0;
        return;
    }
    ct.name[node] = label.substr(0, colon);
    // single precision, as std::stof in the reference parser
    ct.length[node] = static_cast<double>(std::strtof(label.c_str() + colon + 1, nullptr));
}

}  // namespace

bool BPTree::from_newick(const std::string &text, BPTree &out) {
    size_t end = text.size();
    while (end > 0 && (text[end - 1] == ' ' || text[end - 1] == '\t' || text[end - 1] == '\n' ||
                       text[end - 1] == '\r'))
        end--;
    ChildTree ct;
    const uint32_t root = ct.add();
    std::vector<uint32_t> stack;
    uint32_t cur = root;
    std::string label;
    bool in_quote = false;
    for (size_t i = 0; i < end; i++) {
        const char c = text[i];
        if (c == '\n') continue;
        if (c == '\'') {
            in_quote = !in_quote;
            continue;
        }
        if (in_quote) {
            label.push_back(c);
            continue;
        }
        if (c == '(') {
            apply_label(ct, cur, label);
            label.clear();
            stack.push_back(cur);
            cur = ct.add();
            ct.children[stack.back()].push_back(cur);
        } else if (c == ',') {
            apply_label(ct, cur, label);
            label.clear();
            if (stack.empty()) return false;
            cur = ct.add();
            ct.children[stack.back()].push_back(cur);
        } else if (c == ')') {
            apply_label(ct, cur, label);
            label.clear();
            if (stack.empty()) return false;
            cur = stack.back();
            stack.pop_back();
        } else if (c == ';') {
            break;
        } else {
            label.push_back(c);
        }
    }
    apply_label(ct, cur, label);
    if (!stack.empty()) return false;
    out = serialise(ct, root);
    return true;
}

BPTree BPTree::masked(const std::vector<uint8_t> &keep, const std::vector<double> &lengths) const {
    BPTree r;
    r.storage = storage;
    size_t m = 0;
    for (uint8_t k : keep) m += k;
    r.open.resize(m);
    r.length.resize(m);
    r.name.resize(m);
    size_t j = 0;
    for (uint32_t i = 0; i < size(); i++) {
        if (!keep[i]) continue;
        r.open[j] = open[i];
        r.length[j] = lengths[i];
        r.name[j] = name[i];
        j++;
    }
    r.check_parentheses();
    return r;
}

TipMatch BPTree::match_tips(const NameMap &obs, uint32_t n_obs) const {
    TipMatch m;
    const uint32_t n = size();
    m.tags.assign(n, -1);
    m.tree_id = open.data();
    m.tree_size = n;
    // the lookups (read-only on the map, disjoint tags) on up to four host
    // threads for large trees, then the distinct rows counted in one pass
    const unsigned threads = n >= (1u << 16) ? host_threads(4) : 1u;
    const uint32_t span = (n + threads - 1) / threads;
    std::vector<uint8_t> missing(threads, 0);
    parallel_for(threads, threads, [&](unsigned p) {
        const uint32_t lo = p * span, hi = std::min(n ? n - 1 : 0, lo + span);
        bool miss = false;
        for (uint32_t i = lo; i < hi; i++) {
            if (!leaf(i)) continue;
            m.tags[i] = static_cast<int32_t>(obs.find(name[i]));
            miss = miss || m.tags[i] < 0;
        }
        missing[p] = miss ? 1 : 0;
    });
    std::vector<uint8_t> seen(n_obs, 0);
    for (uint32_t i = 0; i + 1 < n; i++) {
        const int32_t row = m.tags[i];
        if (row >= 0 && !seen[row]) {
            seen[row] = 1;
            m.rows_matched++;
        }
    }
    m.all_tips = std::find(missing.begin(), missing.end(), 1) == missing.end();
    return m;
}

BPTree BPTree::shear(const NameSet &keep) const {
    const uint32_t n = size();
    const std::vector<uint32_t> match = partners();
    std::vector<uint8_t> mask(n, 0);
    std::vector<uint32_t> parent(n, UINT32_MAX);
    std::vector<uint32_t> stack;
    for (uint32_t i = 0; i < n; i++) {
        if (open[i]) {
            parent[i] = stack.empty() ? UINT32_MAX : stack.back();
            stack.push_back(i);
        } else if (!stack.empty()) {
            stack.pop_back();
        }
    }
    for (uint32_t i = 0; i + 1 < n; i++) {
        if (!leaf(i) || keep.count(name[i]) == 0) continue;
        mask[i] = mask[i + 1] = 1;
        for (uint32_t p = parent[i]; p != UINT32_MAX && !mask[p]; p = parent[p]) mask[p] = mask[match[p]] = 1;
    }
    return masked(mask, length);
}

BPTree BPTree::collapse() const {
    const uint32_t n = size();
    const std::vector<uint32_t> match = partners();
    std::vector<uint8_t> mask(n, 0);
    std::vector<double> len(length);
    for (uint32_t cur = 0; cur < n; cur++) {  // opening parentheses in index order = preorder
        if (!open[cur]) continue;
        if (leaf(cur) || cur == 0) {
            mask[cur] = mask[match[cur]] = 1;
            continue;
        }
        const uint32_t first = cur + 1;
        const uint32_t last = match[match[cur] - 1];
        if (first == last)
            len[first] = len[first] + len[cur];
        else
            mask[cur] = mask[match[cur]] = 1;
    }
    return masked(mask, len);
}

NameSet BPTree::tip_names() const {
    NameSet out;
    out.reserve(size() / 2 + 1);
    for (uint32_t i = 0; i + 1 < size(); i++)
        if (leaf(i)) out.insert(name[i]);
    return out;
}

uint32_t BPTree::n_tips() const {
    uint32_t c = 0;
    for (uint32_t i = 0; i + 1 < size(); i++) c += leaf(i);
    return c;
}

// Bound by mispredicted branches on the parentheses, so one walk: 31,000 of
// 33,337 tips kept, 1.5 ms; the sheared tree, its flattening, its collapse and
// that one's flattening took 8.1 ms.
FlatTree flatten(const BPTree &t, const std::vector<int32_t> &tags, bool bypass_tips) {
    FlatTree f;
    const uint32_t n = t.size(), most = n / 2;
    f.length.reserve(most);
    f.leaf_obs.reserve(most);
    f.child_ptr.reserve(most + 1);
    f.child_rows.reserve(most);
    f.postorder_row.reserve(most);
    f.leaf_rows.reserve(most / 2 + 1);
    f.parent.reserve(most);
    f.height.reserve(most);
    // with bypassed tips, theirs until the number of embedded rows is known
    std::vector<double> tip_length;
    std::vector<int32_t> tip_obs;
    constexpr uint32_t TIP = 0x80000000u;
    // the lengths of collapsed nodes, lowest first, of the row below them; no
    // other row's come in between, as all else below the chain is dropped
    struct Link {
        uint32_t row;
        double length;
    };
    std::vector<Link> links;

    // One walk over the parentheses: an open node keeps its opening index,
    // the tallest kept child + 1 and where its children start on `pend`, the
    // stack of rows whose parent has not closed yet (left to right).
    struct Open {
        uint32_t o, h, first;
    };
    std::vector<Open> stack;
    stack.reserve(64);
    std::vector<uint32_t> pend;
    pend.reserve(64);
    uint32_t max_height = 0;
    for (uint32_t i = 0; i < n; i++) {
        if (t.open[i]) {
            stack.push_back({i, 0, static_cast<uint32_t>(pend.size())});
            continue;
        }
        if (stack.empty()) continue;
        const Open e = stack.back();
        stack.pop_back();
        if (stack.empty()) break;  // the root closes last, without a row (src/unifrac_cmp.cpp:97-100)
        uint32_t row, h = 0;
        if (e.o + 1 == i) {
            const int32_t obs = tags[e.o];
            if (obs < 0) continue;
            if (bypass_tips) {
                row = TIP | static_cast<uint32_t>(tip_obs.size());
                tip_length.push_back(t.length[e.o]);
                tip_obs.push_back(obs);
            } else {
                row = static_cast<uint32_t>(f.length.size());
                f.length.push_back(t.length[e.o]);
                f.leaf_obs.push_back(obs);
                f.child_ptr.push_back(static_cast<uint32_t>(f.child_rows.size()));
                f.parent.push_back(-1);
                f.height.push_back(0);
            }
            f.leaf_rows.push_back(row);
        } else {
            const uint32_t nk = static_cast<uint32_t>(pend.size()) - e.first;
            if (nk == 0) continue;  // no kept tip below
            if (nk == 1) {          // collapsed into its child, which stays pending
                links.push_back({pend.back(), t.length[e.o]});
                stack.back().h = std::max(stack.back().h, e.h);
                continue;
            }
            row = static_cast<uint32_t>(f.length.size());
            h = e.h;
            f.length.push_back(t.length[e.o]);
            f.leaf_obs.push_back(-1);
            f.child_ptr.push_back(static_cast<uint32_t>(f.child_rows.size()));
            f.child_rows.insert(f.child_rows.end(), pend.begin() + e.first, pend.end());
            if (!bypass_tips)
                for (uint32_t q = e.first; q < pend.size(); q++) f.parent[pend[q]] = static_cast<int32_t>(row);
            f.parent.push_back(-1);
            f.height.push_back(h);
            max_height = std::max(max_height, h);
            pend.resize(e.first);
        }
        f.postorder_row.push_back(row);
        pend.push_back(row);
        stack.back().h = std::max(stack.back().h, h + 1);
    }
    f.n_embedded = static_cast<uint32_t>(f.length.size());
    f.n_nodes = f.n_embedded + static_cast<uint32_t>(tip_obs.size());
    f.child_ptr.resize(f.n_nodes + 1, static_cast<uint32_t>(f.child_rows.size()));
    if (bypass_tips) {
        f.length.insert(f.length.end(), tip_length.begin(), tip_length.end());
        f.leaf_obs.insert(f.leaf_obs.end(), tip_obs.begin(), tip_obs.end());
        f.parent.resize(f.n_nodes, -1);
        f.height.resize(f.n_nodes, 0);
        auto place = [&](uint32_t &row) {
            if (row & TIP) row = f.n_embedded + (row & ~TIP);
        };
        for (uint32_t &r : f.child_rows) place(r);
        for (uint32_t &r : f.postorder_row) place(r);
        for (uint32_t &r : f.leaf_rows) place(r);
        for (Link &l : links) place(l.row);
        for (uint32_t r = 0; r < f.n_embedded; r++)
            for (uint32_t q = f.child_ptr[r]; q < f.child_ptr[r + 1]; q++)
                f.parent[f.child_rows[q]] = static_cast<int32_t>(r);
    }
    // a chain's lengths are added from the top, as in preorder
    for (size_t j = links.size(); j > 0;) {
        const uint32_t row = links[j - 1].row;
        double sum = links[--j].length;
        while (j > 0 && links[j - 1].row == row) sum = links[--j].length + sum;
        f.length[row] += sum;
    }
    // internal rows bucketed by height 1..max_height, rows ascending
    f.level_ptr.assign(max_height + 1, 0);
    for (uint32_t row = 0; row < f.n_embedded; row++)
        if (f.height[row] > 0) f.level_ptr[f.height[row]]++;
    for (uint32_t h = 1; h <= max_height; h++) f.level_ptr[h] += f.level_ptr[h - 1];
    f.level_rows.assign(f.level_ptr[max_height], 0);
    std::vector<uint32_t> fill(f.level_ptr.begin(), f.level_ptr.end());
    for (uint32_t row = 0; row < f.n_embedded; row++)
        if (f.height[row] > 0) f.level_rows[fill[f.height[row] - 1]++] = row;
    return f;
}

uint32_t table_embedded(const FlatTree &f, const std::vector<int32_t> &obs_row, bool bypass_tips,
                        std::vector<uint8_t> *active) {
    std::vector<uint32_t> tips(f.n_nodes, 0);  // kept tips below each row
    uint32_t count = 0;
    if (active) active->assign(f.n_embedded, 0);
    for (uint32_t k = 0; k < f.n_nodes; k++) {
        const uint32_t row = f.postorder_row[k];
        if (f.child_ptr[row] == f.child_ptr[row + 1]) {
            const int32_t o = f.leaf_obs[row];
            const bool kept = o >= 0 && static_cast<size_t>(o) < obs_row.size() && obs_row[o] >= 0;
            tips[row] = kept ? 1 : 0;
            if (kept && !bypass_tips) count++;
            if (active && row < f.n_embedded) (*active)[row] = kept ? 1 : 0;
            continue;
        }
        uint32_t below = 0, kids = 0;
        for (uint32_t q = f.child_ptr[row]; q < f.child_ptr[row + 1]; q++) {
            const uint32_t c = f.child_rows[q];
            below += tips[c];
            kids += tips[c] > 0;
        }
        tips[row] = below;
        if (kids >= 2) count++;
        if (active && row < f.n_embedded) (*active)[row] = below >= (bypass_tips ? 2u : 1u);
    }
    return count;
}

}  // namespace ssu
