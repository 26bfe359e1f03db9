"""The work that users of this UniFrac engine have it do, as cases to measure.

A case is one table (or a batch of tables) with its tree and method, run
through the public Python entry points: device-resident plans (`Plan`,
`BatchPlan`: a program that keeps its table on the GPU and takes the matrix
there), whole calls on host arrays (`one_off_matrix`, `one_off`, `partial`,
`faith_pd`) and the ordination of a matrix on the device (`pcoa_device`).

Trees are random binary trees with Yule clade sizes and exponential branch
lengths; tables have lognormal counts, presence only, or counts rarefied to a
common depth, over features in an order of their own, found equally often or
(as in most surveys) a few of them almost everywhere and the rest rarely.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "unifrac-binaries_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ssu_b200  # noqa: E402
import ssu_synth  # noqa: E402


def listed():
    return [
        # A study of a hundred samples on a small tree, full precision, the
        # table on the GPU: latency and launches count.
        plan("unweighted_fp64_small", "unweighted_fp64", 1000, 128, 0.05),
        # The same study called once from host arrays: the whole call.
        call("weighted_call_small", "matrix", "weighted_normalized_fp64", 1000, 128, 0.05),
        # A large study, weighted normalized in full precision, on the GPU.
        plan("weighted_fp64_2048", "weighted_normalized_fp64", 20000, 2048, 0.01),
        # The same from host arrays to a host matrix.
        call("weighted_call_2048", "matrix", "weighted_normalized_fp64", 20000, 2048, 0.01),
        # Ragged sizes, fp32, weighted unnormalized; features of unequal
        # prevalence, a tenth of the tree's tips not in the table.
        plan("weighted_unnorm_fp32_odd", "weighted_unnormalized", 12345, 1537, 0.02, features=11111, skewed=True),
        # Unweighted in full precision, the default method of many pipelines.
        plan("unweighted_fp64_2048", "unweighted_fp64", 20000, 2048, 0.01),
        # A meta-analysis: 25,000 samples on a 100,000-tip tree, presence
        # only, fp32 - the largest.
        plan("unweighted_fp32_25k", "unweighted", 100000, 25000, 0.005, counts="presence"),
        # Rarefied replicates of one table of 5,000 samples, weighted fp32,
        # as one batch.
        batch("weighted_fp32_replicates", "weighted_normalized", 10000, "replicates", 4, 5000, 5000, 0.02),
        # Independent studies of uneven size on one reference tree, as one
        # batch: generalized UniFrac, and variance adjusted weighted.
        batch("generalized_fp64_uneven", "generalized_fp64", 50000, "uneven", 8, 64, 1024, 0.01, alpha=0.5),
        batch("vaw_fp64_uneven", "weighted_normalized_fp64", 50000, "uneven", 6, 64, 1024, 0.01, vaw=True),
        # Faith's phylogenetic diversity of a large study, from host arrays.
        call("faith_pd_2048", "faith", "faith", 20000, 2048, 0.01),
        # Ordination of a matrix that is on the GPU already.
        {"name": "pcoa_4096", "kind": "pcoa", "samples": 4096, "dims": 10},
    ]


def plan(name, method, tips, samples, density, features=0, counts="lognormal", skewed=False, vaw=False, alpha=1.0):
    return {"name": name, "kind": "plan", "method": method, "tips": tips, "features": features or tips,
            "samples": samples, "density": density, "counts": counts, "skewed": skewed, "vaw": vaw, "alpha": alpha}


def call(name, form, method, tips, samples, density, features=0, counts="lognormal", skewed=False, vaw=False,
         alpha=1.0):
    return dict(plan(name, method, tips, samples, density, features, counts, skewed, vaw, alpha), kind="call",
                form=form)


def batch(name, method, tips, form, tables, lo, hi, density, vaw=False, alpha=1.0):
    return {"name": name, "kind": "batch", "method": method, "tips": tips, "form": form, "tables": tables, "lo": lo,
            "hi": hi, "density": density, "vaw": vaw, "alpha": alpha}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: single tables of 9 to 4,096 samples on trees of 300 to
    50,000 tips with every method, precision and option, larger presence
    tables on the fp32 unweighted path, batches, whole calls, ordinations."""
    pick = rng.random()
    methods = ["unweighted", "weighted_normalized", "weighted_unnormalized", "generalized"]
    if pick < 0.08:
        return {"kind": "pcoa", "samples": _log(rng, 64, 4096), "dims": rng.randint(2, 16)}
    if pick < 0.18:
        return {k: v for k, v in plan("", "unweighted", _log(rng, 5000, 60000), _log(rng, 3000, 12000),
                                      math.exp(rng.uniform(math.log(0.002), math.log(0.02))),
                                      counts="presence").items() if k != "name"}
    method = rng.choice(methods)
    vaw = rng.random() < 0.25
    alpha = rng.choice([0.0, 0.25, 0.5, 1.0, 1.5]) if method == "generalized" else 1.0
    method += rng.choice(["", "_fp64"])
    density = math.exp(rng.uniform(math.log(0.004), math.log(0.06)))
    if pick < 0.38:
        if rng.random() < 0.4:
            heavy = vaw or method.startswith("generalized")
            n = _log(rng, 200, 1200 if heavy else 5000)
            c = batch("", method, _log(rng, 1000, 10000), "replicates", rng.randint(2, 4), n, n, density, vaw, alpha)
        else:
            c = batch("", method, _log(rng, 2000, 50000), "uneven", rng.randint(2, 8), _log(rng, 16, 80),
                      _log(rng, 200, 1024), min(density, 0.02), vaw, alpha)
    else:
        heavy = vaw or method.startswith("generalized")
        tips = _log(rng, 300, 50000)
        most = max(64, min(1400 if heavy else 4096, int(math.sqrt((2e10 if heavy else 1e11) / tips))))
        samples = _log(rng, 9, most)
        args = (tips, samples, density, int(tips * rng.choice([1.0, 0.93, 0.7])), "lognormal", rng.random() < 0.5,
                vaw, alpha)
        if pick < 0.8:
            c = plan("", method, *args)
        else:
            c = call("", rng.choice(["matrix", "matrix", "condensed", "stripes", "faith"]), method, *args)
    c.pop("name")
    return c


# ------------------------------------------------------------------- inputs

def _yule_tree(rng, tips):
    """A random binary tree, each clade of m tips split uniformly in two:
    per node (preorder rows) the span [a, b) of its tips and the position of
    its opening parenthesis."""
    spans, opens = [], []
    a, b, at = np.array([0]), np.array([tips]), np.array([0])
    while len(a):
        spans.append((a, b))
        opens.append(at)
        inner = b - a > 1
        a, b, at = a[inner], b[inner], at[inner]
        left = 1 + np.floor(rng.random(len(a)) * (b - a - 1)).astype(np.int64)
        mid = a + left
        at2 = at + 1 + 2 * (2 * left - 1)
        a, b, at = np.concatenate([a, mid]), np.concatenate([mid, b]), np.concatenate([at + 1, at2])
    a = np.concatenate([s[0] for s in spans])
    b = np.concatenate([s[1] for s in spans])
    at = np.concatenate(opens)
    order = np.argsort(at)
    return a[order], b[order], at[order]


def _tree(rng, tips):
    """(BPTree, first tip, end tip, length of every node but the root)."""
    a, b, at = _yule_tree(rng, tips)
    n = 2 * (2 * tips - 1)
    structure = np.zeros(n, dtype=bool)
    structure[at] = True
    lengths = np.zeros(n)
    node_len = rng.exponential(0.05, size=len(at))
    node_len[0] = 0.0
    lengths[at] = node_len
    names = [""] * n
    leaf = b - a == 1
    for pos, tip in zip(at[leaf].tolist(), a[leaf].tolist()):
        names[pos] = "T%d" % tip
    return ssu_synth.BPTree(structure, lengths, names), a[1:], b[1:], node_len[1:]


def _csr(flat, values, tip_of_feature, samples):
    """(Table, tip of each feature) from sorted cells feature * samples + sample."""
    feature, sample = np.divmod(flat, samples)
    indptr = np.zeros(len(tip_of_feature) + 1, dtype=np.uint32)
    indptr[1:] = np.cumsum(np.bincount(feature, minlength=len(tip_of_feature)))
    return ssu_synth.Table(["T%d" % t for t in tip_of_feature.tolist()], ["S%d" % j for j in range(samples)], indptr,
                           sample.astype(np.uint32), values.astype(np.float64))


def _cells(gen, features, samples, density, skewed, presence):
    """Distinct cells of a table, sorted: each sample with about
    density * features of its features."""
    dev = gen.device
    rich = torch.full((samples,), density * features, device=dev)
    if presence:  # richness spread log-uniformly over a factor of 40
        rich = torch.exp(torch.rand(samples, generator=gen, device=dev) * math.log(40.0)) * (
            density * features * math.log(40.0) / 39.0)
    rich = rich.round().long().clamp(1, features)
    sample = torch.repeat_interleave(torch.arange(samples, device=dev), rich)
    u = torch.rand(len(sample), generator=gen, device=dev, dtype=torch.float64)
    feature = ((u ** 3 if skewed else u) * features).long().clamp(0, features - 1)
    return torch.unique(feature * samples + sample)


def _counts(gen, cells, kind):
    if kind == "presence":
        return torch.ones(len(cells), device=gen.device, dtype=torch.float64)
    z = torch.randn(len(cells), generator=gen, device=gen.device, dtype=torch.float64)
    return torch.exp(2.0 + 1.5 * z).round() + 1.0


def _table(gen, tip_of_feature, samples, density, skewed, counts):
    cells = _cells(gen, len(tip_of_feature), samples, density, skewed, counts == "presence")
    values = _counts(gen, cells, counts)
    return _csr(cells.cpu().numpy(), values.cpu().numpy(), tip_of_feature, samples), tip_of_feature


def _replicates(gen, tip_of_feature, samples, density, count, depth=1000):
    """`count` draws of `depth` reads of each sample, without replacement, of
    one table, its features kept."""
    dev = gen.device
    cells = _cells(gen, len(tip_of_feature), samples, density, False, False)
    reads = (_counts(gen, cells, "lognormal") * 3).long()
    # every sample reaches the depth: the missing reads go to its first cell
    sample = cells % samples
    total = torch.zeros(samples, dtype=torch.long, device=dev).index_add_(0, sample, reads)
    first = torch.full((samples,), len(cells), dtype=torch.long, device=dev).scatter_reduce_(
        0, sample, torch.arange(len(cells), device=dev), "amin")
    has = first < len(cells)
    reads[first[has]] += (depth - total[has]).clamp(min=0)
    unit = torch.repeat_interleave(torch.arange(len(cells), device=dev), reads)
    out = []
    for _ in range(count):
        key = sample[unit] * (1 << 40) + torch.randint(1 << 40, (len(unit),), generator=gen, device=dev)
        order = torch.argsort(key)
        s = sample[unit[order]]
        start = torch.searchsorted(s, torch.arange(samples, device=dev))
        kept = unit[order][torch.arange(len(s), device=dev) - start[s] < depth]
        values = torch.bincount(kept, minlength=len(cells))
        on = values > 0
        out.append((_csr(cells[on].cpu().numpy(), values[on].cpu().numpy(), tip_of_feature, samples), tip_of_feature))
    return out


def _sizes(case):
    n, lo, hi = case["tables"], case["lo"], case["hi"]
    return [int(round(lo * (hi / lo) ** ((t + 0.5) / n))) for t in range(n)]


def _inputs(case, seed):
    """Tree, the spans and lengths of its nodes, and [(table, tips)].  The
    tree, and which of its tips are features, go by the tree's size alone
    (studies share a reference tree); the tables are the seed's."""
    tips = case["tips"]
    rng = np.random.default_rng(tips)
    tree, a, b, length = _tree(rng, tips)
    tip_of_feature = rng.permutation(tips)[:case.get("features", tips)]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["kind"] != "batch":
        tables = [_table(gen, tip_of_feature, case["samples"], case["density"], case["skewed"], case["counts"])]
    elif case["form"] == "replicates":
        tables = _replicates(gen, tip_of_feature, case["lo"], case["density"], case["tables"])
    else:
        tables = [_table(gen, tip_of_feature, n, case["density"], False, "lognormal") for n in _sizes(case)]
    return tree, (a, b, length), tables


def _points(case, seed):
    """A distance matrix with the falling spectrum of real ordinations:
    distances of points whose spread falls by a factor of 0.75 an axis."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    x = torch.randn(case["samples"], 48, generator=gen, device="cuda", dtype=torch.float64)
    x = x * 0.75 ** torch.arange(48, device="cuda", dtype=torch.float64)
    d2 = (x * x).sum(1)
    d = (d2[:, None] + d2[None, :] - 2 * (x @ x.T)).clamp(min=0).sqrt()
    d = (d + d.T) / (2 * d.max())
    return d.fill_diagonal_(0.0).contiguous()


# --------------------------------------------------------------------- runs

class _DeviceArray:
    """A plan's result in device memory, for torch to look at in place."""

    def __init__(self, owner, pointer, shape, dtype):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": dtype, "data": (pointer, False), "version": 3}


_STREAM = []


def _stream():
    """The program's one stream, on which all its plans run in turn."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0]


def prepare(case, seed):
    if case["kind"] == "pcoa":
        return {"case": case, "matrix": _points(case, seed)}
    tree, _, tables = _inputs(case, seed)
    tables = [t for t, _ in tables]
    if case["kind"] == "call":
        return {"case": case, "tree": tree, "table": tables[0]}
    options = {"variance_adjust": case["vaw"], "alpha": case["alpha"]}
    if case["kind"] == "plan":
        p = ssu_b200.Plan(tree, tables[0], case["method"], **options)
        sizes, offsets = [p.n], [0]
    else:
        p = ssu_b200.BatchPlan(tree, tables, case["method"], **options)
        sizes, offsets = p.sizes, p.offsets
    kind, width = ("<f8", 8) if case["method"].endswith("_fp64") else ("<f4", 4)
    out = [torch.as_tensor(_DeviceArray(p, p.device_result() + o * width, (n, n), kind), device="cuda")
           for n, o in zip(sizes, offsets)]
    return {"case": case, "plan": p, "out": out, "stream": _stream().cuda_stream}


def run(state):
    case = state["case"]
    if case["kind"] == "pcoa":
        values, samples, explained = ssu_b200.pcoa_device(state["matrix"].data_ptr(), case["samples"], case["dims"])
        return {"eigenvalues": values, "samples": samples, "explained": explained}
    if case["kind"] == "call":
        tree, table = state["tree"], state["table"]
        if case["form"] == "faith":
            return ssu_b200.faith_pd(tree, table)[0]
        options = {"variance_adjust": case["vaw"], "alpha": case["alpha"]}
        if case["form"] == "matrix":
            return ssu_b200.one_off_matrix(tree, table, case["method"], copy=False, **options)[0]
        if case["form"] == "condensed":
            return ssu_b200.one_off(tree, table, case["method"], **options)[0]
        return ssu_b200.partial(tree, table, case["method"], *_window(case), **options)[0]
    state["plan"].execute(state["stream"])
    return state["out"]


def _window(case):
    """The first half of the stripes: one of two jobs that share a matrix."""
    return 0, max(1, (case["samples"] + 1) // 4)


# --------------------------------------------------------------------- work

def _branches(tips, density, pairwise):
    """Expected branches of a Yule tree with a read in one sample (of either
    of two, `pairwise`): 2 T / (m (m + 1)) clades of m tips."""
    m = np.arange(1, tips)
    clades = np.where(m == 1, float(tips), 2.0 * tips / (m * (m + 1.0)))
    return float((clades * (1.0 - (1.0 - density) ** (m * (2.0 if pairwise else 1.0)))).sum())


def work(case):
    """The table and tree read once, the result written once; one multiply
    and add for each branch that one or both samples of a pair have."""
    if case["kind"] == "pcoa":
        n, d = case["samples"], case["dims"]
        return {"bytes": 8.0 * n * n + 8.0 * n * d, "flops": 4.0 * n * n * (d + 10) * 2}
    if case["kind"] == "batch":
        sizes = _sizes(case) if case["form"] == "uneven" else [case["lo"]] * case["tables"]
    else:
        sizes = [case["samples"]]
    tips, density = case["tips"], case["density"]
    cells = sum(sizes) * density * case.get("features", tips)
    width = 8.0 if case["method"].endswith("_fp64") else 4.0
    read = 12.0 * cells + 4.0 * tips * len(sizes) + 9.0 * 4 * tips
    if case.get("form") == "faith":
        return {"bytes": read + 8.0 * sizes[0], "flops": 2.0 * sizes[0] * _branches(tips, density, False)}
    pairs = sum(n * (n - 1) / 2.0 for n in sizes)
    out = {"condensed": 8.0 * pairs, "stripes": 4.0 * pairs}.get(case.get("form"), width * sum(n * n for n in sizes))
    return {"bytes": read + out, "flops": 2.0 * pairs * _branches(tips, density, True)}


# -------------------------------------------------------------------- exact

def exact(case, seed):
    if case["kind"] == "pcoa":
        return _exact_pcoa(_points(case, seed), case["dims"])
    _, (a, b, length), tables = _inputs(case, seed)
    a, b = (torch.from_numpy(x).cuda() for x in (a, b))
    length = torch.from_numpy(length).cuda()
    faith = case.get("form") == "faith"
    out = []
    for table, tip in tables:
        n = table.n_samples
        if n * n * len(length) > (1.3e14 if case["method"].startswith("unweighted") and not case["vaw"] else 6e11):
            return None
        cum = _cumulated(table, tip, case["tips"])
        if faith:
            s = torch.zeros(n, dtype=torch.float64, device="cuda")
            for c in _chunks(len(length), n):
                s += (length[c, None] * (cum[b[c]] > cum[a[c]])).sum(0)
            return s.cpu().numpy()
        d = _exact_matrix(case, cum, a, b, length).fill_diagonal_(0.0)
        out.append(d)
    if case["kind"] == "call":
        d = out[0]
        n = d.shape[0]
        if case["form"] == "condensed":
            k, l = torch.triu_indices(n, n, 1, device="cuda")
            return d[k, l].cpu().numpy()
        if case["form"] == "stripes":
            first, last = _window(case)
            k = torch.arange(n, device="cuda")
            return torch.stack([d[k, (k + s + 1) % n] for s in range(first, last)]).cpu().numpy()
        return d.cpu().numpy()
    return out


def _cumulated(table, tip, tips):
    """Reads of the first t tips, [tips + 1][samples]: whole numbers, exact."""
    dtype = torch.int32 if table.n_samples > 4096 else torch.float64
    n = table.n_samples
    cum = torch.zeros(tips + 1, n, dtype=dtype, device="cuda")
    feature = np.repeat(np.arange(table.n_obs), np.diff(table.indptr.astype(np.int64)))
    row = torch.from_numpy(tip[feature].astype(np.int64) + 1).cuda()
    col = torch.from_numpy(table.indices.astype(np.int64)).cuda()
    cum[row, col] = torch.from_numpy(table.data).cuda().to(dtype)
    return torch.cumsum(cum, 0, dtype=dtype)


def _chunks(nodes, per_node, room=1 << 27):
    step = max(1, room // max(1, per_node))
    return [slice(i, min(nodes, i + step)) for i in range(0, nodes, step)]


def _exact_matrix(case, cum, a, b, length):
    n = cum.shape[1]
    method = case["method"].replace("_fp64", "")
    total = cum[-1].double()
    f64 = {"dtype": torch.float64, "device": "cuda"}
    num, den = torch.zeros(n, n, **f64), torch.zeros(n, n, **f64)
    if case["vaw"] or method == "generalized":
        m = total[:, None] + total[None, :]
        alpha = case["alpha"]
        for c in _chunks(len(length), n * n):
            x = cum[b[c]] - cum[a[c]]
            keep = (x > 0).any(1)
            x, L = x[keep], length[c][keep, None, None]
            u = x / total
            s, d = u[:, :, None] + u[:, None, :], (u[:, :, None] - u[:, None, :]).abs()
            on = s > 0
            if case["vaw"]:
                mi = x[:, :, None] + x[:, None, :]
                v = mi * (m - mi)
                on = v > 0
                v = torch.where(on, v.clamp(min=0).sqrt(), torch.ones_like(v))
                s, d = s / v, d / v
            if method == "generalized":
                p = torch.where(on, s, torch.ones_like(s)) ** alpha * L
                d = p * torch.where(on, d / torch.where(on, s, torch.ones_like(s)), torch.zeros_like(d))
                s = p
            elif method == "unweighted":
                h = (x > 0).double()
                either, one = (h[:, :, None] + h[:, None, :]) > 0, h[:, :, None] != h[:, None, :]
                s, d = either * L / v, one * L / v
            else:
                s, d = s * L, d * L
            num += torch.where(on, d, torch.zeros_like(d)).sum(0)
            den += torch.where(on, s, torch.zeros_like(s)).sum(0)
        return num if method == "weighted_unnormalized" else num / den
    r = torch.zeros(n, **f64)
    for c in _chunks(len(length), n):
        x = cum[b[c]] - cum[a[c]]
        L = length[c, None]
        if method == "unweighted":
            h = (x > 0).double()
            r += (h * L).sum(0)
            num += (h * L).T @ h
        else:
            u = x / total
            r += (u * L).sum(0)
            y = (u * L).T.contiguous()
            num += torch.cdist(y, y, p=1.0)
    if method == "unweighted":
        den = r[:, None] + r[None, :] - num
        return (den - num) / den
    return num if method == "weighted_unnormalized" else num / (r[:, None] + r[None, :])


def _exact_pcoa(d, dims):
    n = d.shape[0]
    e = -0.5 * d * d
    mean = e.mean(0)
    f = e - mean[:, None] - mean[None, :] + mean.mean()
    w, v = torch.linalg.eigh(f)
    w, v = w.flip(0), v.flip(1)
    k = min(dims, n)
    top = v[:, :k]
    sign = torch.sign(top.gather(0, top.abs().argmax(0, keepdim=True)))
    samples = top * sign * w[:k].clamp(min=0).sqrt()
    return {"eigenvalues": w[:k].cpu().numpy(), "samples": samples.cpu().numpy(),
            "explained": (w[:k] / torch.trace(f)).cpu().numpy()}
