"""Parity of the CUDA path (through the C ABI of libssu_b200.so) with the
oracle, on seeded inputs.

Bars: fp64 methods within 1e-12 relative of the oracle (1e-13 absolute where
the oracle value is 0); fp32 methods within 4x the reference fp32 build's own
error against fp64 on the same input (measured with the oracle's fp32 mode),
floored at 1e-6; NaN patterns identical."""
import os

import numpy as np
import pytest

import ssu_synth
from conftest import ROOT, matrix_from_stripes, rel_err, stripes_from_golden

pytestmark = pytest.mark.gpu

METHODS = ["unweighted", "unweighted_unnormalized", "weighted_normalized", "weighted_unnormalized", "generalized"]
FP64_REL = 1e-12
FP64_ABS = 1e-13


def _case(seed, n_tips=90, n_samples=37, density=0.12, drop=7):
    tree = ssu_synth.random_binary_tree(n_tips, 0.1, seed)
    table = ssu_synth.geometric_table(tree.tip_names()[: n_tips - drop], n_samples, density, 10.0, seed + 3)
    return tree, table


def check_fp64(gpu, ref):
    r, z = rel_err(gpu, ref)
    assert r <= FP64_REL, f"max rel err {r:.3e}"
    assert z <= FP64_ABS, f"max abs err at zeros {z:.3e}"


def check_fp32(gpu32, oracle, tree, table, method, **kw):
    o64 = oracle.oracle_one_off(tree, table, method + "_fp64", **kw)["matrix"]
    o32 = oracle.oracle_one_off(tree, table, method + "_fp32", **kw)["matrix"]
    ref_err, ref_zero = rel_err(o32, o64)
    ours, ours_zero = rel_err(gpu32, o64)
    assert ours <= max(4 * ref_err, 1e-6), (ours, ref_err)
    assert ours_zero <= max(4 * ref_zero, 1e-6)


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("vaw", [False, True])
@pytest.mark.parametrize("bypass", [False, True])
def test_fp64_matches_oracle(ssu, oracle_mod, method, vaw, bypass):
    tree, table = _case(21)
    kw = dict(variance_adjust=vaw, bypass_tips=bypass, alpha=0.5)
    gpu, ids = ssu.one_off_matrix(tree, table, method + "_fp64", **kw)
    assert ids == table.sample_ids
    check_fp64(gpu, oracle_mod.oracle_one_off(tree, table, method + "_fp64", **kw)["matrix"])


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("vaw", [False, True])
def test_fp32_within_reference_fp32_error(ssu, oracle_mod, method, vaw):
    tree, table = _case(22)
    kw = dict(variance_adjust=vaw, alpha=0.5)
    gpu, _ = ssu.one_off_matrix(tree, table, method + "_fp32", **kw)
    assert gpu.dtype == np.float32
    check_fp32(gpu, oracle_mod, tree, table, method, **kw)


@pytest.mark.parametrize("alpha", [0.0, 0.25, 0.5, 1.0, 1.5])
def test_generalized_alphas(ssu, oracle_mod, alpha):
    tree, table = _case(23)
    for vaw in (False, True):
        gpu, _ = ssu.one_off_matrix(tree, table, "generalized_fp64", variance_adjust=vaw, alpha=alpha)
        check_fp64(gpu, oracle_mod.oracle_one_off(tree, table, "generalized_fp64", variance_adjust=vaw,
                                                  alpha=alpha)["matrix"])


@pytest.mark.parametrize("n", [2, 3, 5, 63, 64, 65, 127, 128, 129, 200, 255, 256, 257])
@pytest.mark.parametrize("method", ["unweighted_fp64", "weighted_normalized_fp64", "generalized_fp64"])
def test_tile_boundaries(ssu, oracle_mod, n, method):
    tree, table = _case(100 + n, n_tips=70, n_samples=n, density=0.2, drop=0)
    gpu, _ = ssu.one_off_matrix(tree, table, method, alpha=0.5)
    check_fp64(gpu, oracle_mod.oracle_one_off(tree, table, method, alpha=0.5)["matrix"])
    assert np.all(np.diag(gpu) == 0)
    np.testing.assert_array_equal(gpu, gpu.T)


GOLDEN_CASES = [
    ("test_unweighted_unifrac", "", "unweighted_fp64", {}),
    ("test_unweighted_unifrac", "", "unweighted_fp32", {}),
    ("test_unweighted_unifrac_fast", "", "unweighted_fp64", {"bypass_tips": True}),
    ("test_unnormalized_unweighted_unifrac", "", "unweighted_unnormalized_fp64", {}),
    ("test_unnormalized_weighted_unifrac", "", "weighted_unnormalized_fp64", {}),
    ("test_normalized_weighted_unifrac", "", "weighted_normalized_fp64", {}),
    ("test_normalized_weighted_unifrac", "", "weighted_normalized_fp32", {}),
    ("test_generalized_unifrac", "w_", "generalized_fp64", {"alpha": 1.0}),
    ("test_generalized_unifrac", "d0_", "generalized_fp64", {"alpha": 0.0}),
    ("test_generalized_unifrac", "d05_", "generalized_fp64", {"alpha": 0.5}),
    ("test_vaw_unifrac_weighted_normalized", "w_", "weighted_normalized_fp64", {"variance_adjust": True}),
]


@pytest.mark.parametrize("func,prefix,method,kw", GOLDEN_CASES)
def test_reference_goldens_through_c_abi(ssu, golden, test_tree, test_table, func, prefix, method, kw):
    exp = stripes_from_golden(golden["test_su"][func], prefix)
    gpu, _ = ssu.one_off_matrix(test_tree, test_table, method, **kw)
    np.testing.assert_allclose(gpu, matrix_from_stripes(exp, 6), atol=1e-6, rtol=0)
    stripes, meta = ssu.partial(test_tree, test_table, method, 0, 3, **kw)
    np.testing.assert_allclose(stripes, exp, atol=1e-6, rtol=0)
    assert meta["total"] == 3 and meta["upper"]


def test_faith_goldens_through_c_abi(ssu, golden, test_table):
    exp = golden["test_su"]["test_faith_pd"]["arrays"]["exp"][0]
    for tre in ("test_faith.tre", "test_faith_shear.tre"):
        tree = ssu_synth.parse_newick(golden["trees"][tre])
        vals, ids = ssu.faith_pd(tree, test_table)
        np.testing.assert_allclose(vals, exp, atol=1e-6, rtol=0)
        assert ids == test_table.sample_ids


@pytest.mark.parametrize("n", [6, 7, 40, 41, 300])
def test_partial_windows_and_condensed(ssu, oracle_mod, n):
    tree, table = _case(40 + n, n_tips=80, n_samples=n, density=0.2, drop=0)
    method = "weighted_normalized_fp64"
    s_total = (n + 1) // 2
    windows = [(0, s_total), (0, 1), (s_total - 1, s_total), (s_total // 3, max(s_total // 3 + 1, 2 * s_total // 3))]
    for start, stop in windows:
        gpu, meta = ssu.partial(tree, table, method, start, stop)
        ref = oracle_mod.oracle_one_off(tree, table, method, stripe_start=start, stripe_stop=stop)["stripes"]
        check_fp64(gpu, ref)
        assert (meta["start"], meta["stop"], meta["total"]) == (start, stop, s_total)
    cf, ids, upper = ssu.one_off(tree, table, method)
    full = oracle_mod.oracle_one_off(tree, table, method)["matrix"]
    iu = np.triu_indices(n, 1)
    check_fp64(cf, full[iu])
    assert upper and len(cf) == n * (n - 1) // 2


def test_partial_out_of_range_is_an_error_not_an_exit(ssu, test_tree, test_table):
    with pytest.raises(ssu.SSUError) as e:
        ssu.partial(test_tree, test_table, "unweighted_fp64", 0, 4)
    assert e.value.status == 6


def test_faith_filters_empty_samples(ssu, oracle_mod):
    tree, table = _case(51, n_samples=30)
    dense = table.dense()
    dense[:, [0, 7]] = 0
    flat = np.flatnonzero(dense.ravel() > 0)
    t2 = ssu_synth.make_table(table.obs_ids, table.n_samples, flat, dense.ravel()[flat])
    vals, ids = ssu.faith_pd(tree, t2)
    ref = oracle_mod.oracle_faith_pd(tree, t2)
    assert ids == [t2.sample_ids[i] for i in ref["kept"]]
    np.testing.assert_allclose(vals, ref["values"], rtol=1e-12, atol=0)


def test_empty_samples_give_reference_nan_pattern(ssu, oracle_mod):
    tree, table = _case(52, n_samples=20)
    dense = table.dense()
    dense[:, [3, 4]] = 0
    flat = np.flatnonzero(dense.ravel() > 0)
    t2 = ssu_synth.make_table(table.obs_ids, table.n_samples, flat, dense.ravel()[flat])
    for m in METHODS:
        gpu, _ = ssu.one_off_matrix(tree, t2, m + "_fp64", alpha=0.5)
        ref = oracle_mod.oracle_one_off(tree, t2, m + "_fp64", alpha=0.5)["matrix"]
        assert np.array_equal(np.isnan(gpu), np.isnan(ref)), m
        check_fp64(gpu, ref)


def test_dense_pair(ssu, golden, oracle_mod):
    tree = ssu_synth.parse_newick(golden["trees"]["test.tre"])
    obs = ["GG_OTU_1", "GG_OTU_2", "GG_OTU_3", "GG_OTU_4", "GG_OTU_5"]
    s1, s3 = [0, 5, 0, 2, 0], [1, 0, 1, 1, 1]
    d = ssu.dense_pair(tree, obs, s1, s3, "unweighted_fp64")
    flat = [i * 2 + j for i in range(5) for j, v in enumerate((s1[i], s3[i])) if v > 0]
    vals = [(s1, s3)[f % 2][f // 2] for f in flat]
    t = ssu_synth.make_table(obs, 2, np.array(flat), np.array(vals, dtype=float))
    exp = oracle_mod.oracle_one_off(tree, t, "unweighted_fp64")["matrix"][0, 1]
    assert abs(d - exp) <= 1e-12 * abs(exp)
    d32 = ssu.dense_pair(tree, obs, s1, s3, "unweighted")
    assert abs(d32 - 0.57142857) < 1e-6  # test/capi_inmem_test.c exp13


def test_unnormalized_sample_counts(ssu, oracle_mod):
    tree, table = _case(53)
    for m in ("weighted_unnormalized_fp64", "weighted_normalized_fp64", "generalized_fp64"):
        gpu, _ = ssu.one_off_matrix(tree, table, m, normalize=False, alpha=0.5)
        check_fp64(gpu, oracle_mod.oracle_one_off(tree, table, m, normalize=False, alpha=0.5)["matrix"])


def test_plan_api_matches_one_off(ssu):
    tree, table = _case(54, n_samples=150)
    for m in ("weighted_normalized_fp64", "unweighted_fp32"):
        plan = ssu.Plan(tree, table, m)
        plan.set_timing(True)
        plan.execute()
        out = plan.result()
        e, p, f = plan.stage_ms()
        assert p > 0 and e >= 0
        ref, _ = ssu.one_off_matrix(tree, table, m)
        np.testing.assert_array_equal(out, ref)
        assert plan.work_units() == 150 * 149 // 2 * plan.n_embedded()
        assert plan.launches() >= 2
        plan.close()


def test_mmap_backed_result(ssu, tmp_path):
    tree, table = _case(55)
    a, _ = ssu.one_off_matrix(tree, table, "weighted_unnormalized_fp64", mmap_dir=str(tmp_path))
    b, _ = ssu.one_off_matrix(tree, table, "weighted_unnormalized_fp64")
    np.testing.assert_array_equal(a, b)


def test_rarefaction_keeps_deep_samples(ssu):
    tree, table = _case(56, n_samples=25, density=0.5)
    totals = table.dense().sum(axis=0)
    depth = int(np.percentile(totals, 40))
    ssu.lib().ssu_set_random_seed(7)
    m, ids = ssu.one_off_matrix(tree, table, "unweighted_fp64", subsample_depth=depth)
    keep = [table.sample_ids[j] for j in range(table.n_samples) if totals[j] >= depth]
    assert ids == keep
    assert m.shape == (len(keep), len(keep))
    assert np.all(np.isfinite(m))


def test_20k_tips_2048_samples_full_size_stripe_windows(ssu, oracle_mod):
    """Full 20,000-tip x 2,048-sample input: the GPU matrix against
    the oracle on the first and last stripes, plus matrix properties."""
    tree, table = ssu_synth.lognormal_20k_tips_2048_samples()
    n = table.n_samples
    s_total = (n + 1) // 2
    for m in ("weighted_normalized_fp64", "weighted_unnormalized_fp64"):
        gpu, _ = ssu.one_off_matrix(tree, table, m)
        assert np.all(np.diag(gpu) == 0)
        np.testing.assert_array_equal(gpu, gpu.T)
        assert np.all(np.isfinite(gpu))
        for start, stop in [(0, 2), (s_total - 2, s_total)]:
            ref = oracle_mod.oracle_one_off(tree, table, m, stripe_start=start, stripe_stop=stop)["stripes"]
            got = np.array([[gpu[k, (k + s + 1) % n] for k in range(n)] for s in range(start, stop)])
            check_fp64(got, ref)
    gpu32, _ = ssu.one_off_matrix(tree, table, "weighted_normalized_fp32")
    ref = oracle_mod.oracle_one_off(tree, table, "weighted_normalized_fp64", stripe_start=0, stripe_stop=1)["stripes"]
    got = np.array([gpu32[k, (k + 1) % n] for k in range(n)], dtype=np.float64)
    r, _ = rel_err(got, ref[0])
    assert r < 1e-4


def test_zero_copy_result_view_outlives_its_parent(ssu):
    import gc
    tree, table = _case(57, n_samples=64)
    ref, _ = ssu.one_off_matrix(tree, table, "weighted_normalized_fp64")
    view, _ = ssu.one_off_matrix(tree, table, "weighted_normalized_fp64", copy=False)
    row = view[3]
    del view
    gc.collect()
    np.testing.assert_array_equal(row, ref[3])
    v32, _ = ssu.one_off_matrix(tree, table, "weighted_normalized_fp32", copy=False)
    assert v32.dtype == np.float32 and v32.shape == (64, 64)


def test_marshalled_inputs_follow_replaced_arrays(ssu):
    tree, table = _case(58, n_samples=40)
    other = ssu_synth.geometric_table(table.obs_ids, 40, 0.12, 10.0, 991)
    first, _ = ssu.one_off_matrix(tree, table, "weighted_unnormalized_fp64")
    again, _ = ssu.one_off_matrix(tree, table, "weighted_unnormalized_fp64")
    np.testing.assert_array_equal(first, again)
    table.indptr, table.indices, table.data = other.indptr, other.indices, other.data
    swapped, _ = ssu.one_off_matrix(tree, table, "weighted_unnormalized_fp64")
    ref, _ = ssu.one_off_matrix(tree, other, "weighted_unnormalized_fp64")
    np.testing.assert_array_equal(swapped, ref)
    table.data = other.data.copy()
    plain, _ = ssu.one_off_matrix(tree, table, "weighted_unnormalized_fp64", normalize=False)
    table.data *= 3.0  # in place: the marshalled view shares the array
    tripled, _ = ssu.one_off_matrix(tree, table, "weighted_unnormalized_fp64", normalize=False)
    np.testing.assert_allclose(tripled, 3.0 * plain, rtol=1e-12)


def _near_duplicates(seed, n_tips=150, n_base=12, copies=4):
    """Samples in clusters of near-duplicates: copies of a base sample with
    one count nudged by a relative 1e-7 (or not at all), so the weighted
    distances inside a cluster are tiny or exactly zero."""
    tree = ssu_synth.random_binary_tree(n_tips, 0.1, seed)
    base = ssu_synth.geometric_table(tree.tip_names(), n_base, 0.1, 10.0, seed + 1).dense()
    base[0, :] += 1.0  # no empty sample
    rng = np.random.default_rng(seed + 2)
    cols = []
    for j in range(n_base):
        for c in range(copies):
            col = base[:, j].copy()
            if c:
                nz = np.flatnonzero(col)
                col[nz[rng.integers(0, nz.size)]] *= 1.0 + 1e-7 * c
            cols.append(col)
    dense = np.stack(cols, axis=1)
    flat = np.flatnonzero(dense.ravel() > 0)
    table = ssu_synth.make_table(tree.tip_names(), dense.shape[1], flat, dense.ravel()[flat])
    return tree, table


@pytest.mark.parametrize("method", ["weighted_normalized_fp64", "weighted_unnormalized_fp64"])
def test_weighted_close_pairs_are_exact(ssu, oracle_mod, method):
    """Pairs whose sparse-form subtraction could lose digits are recomputed
    in the exact |u - v| form: near-duplicate samples still meet 1e-12."""
    tree, table = _near_duplicates(61)
    gpu, _ = ssu.one_off_matrix(tree, table, method)
    ref = oracle_mod.oracle_one_off(tree, table, method)["matrix"]
    check_fp64(gpu, ref)
    small = (ref > 0) & (ref < 1e-5)
    assert small.any()


@pytest.mark.parametrize("method", ["weighted_normalized", "weighted_unnormalized"])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_weighted_sparse_and_dense_forms_agree(ssu, monkeypatch, method, prec):
    tree, table = _case(62, n_tips=300, n_samples=300, density=0.03)
    hybrid, _ = ssu.one_off_matrix(tree, table, f"{method}_{prec}")
    monkeypatch.setenv("UNIFRAC_B200_WEIGHTED_MODE", "dense")
    dense, _ = ssu.one_off_matrix(tree, table, f"{method}_{prec}")
    if prec == "fp64":
        check_fp64(hybrid, dense)
    else:
        np.testing.assert_allclose(hybrid, dense, rtol=5e-6, atol=1e-7)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("method", ["weighted_normalized", "weighted_unnormalized"])
def test_weighted_pair_scatter_and_tile_walk_agree(ssu, monkeypatch, method, prec):
    """The sparse rows as per-pair fixed-point sums (the default) against the
    tile kernel's own walk: the same to fp64 rounding, and the integer sums
    make repeated calls agree bit for bit in both precisions."""
    tree, table = _case(65, n_tips=500, n_samples=700, density=0.02)
    scatter = [ssu.one_off_matrix(tree, table, f"{method}_{prec}")[0] for _ in range(2)]
    np.testing.assert_array_equal(scatter[0], scatter[1])
    monkeypatch.setenv("UNIFRAC_B200_HYBRID_SCATTER", "0")
    monkeypatch.setenv("UNIFRAC_B200_DETERMINISTIC", "1")
    walk, _ = ssu.one_off_matrix(tree, table, f"{method}_{prec}")
    if prec == "fp64":
        check_fp64(scatter[0], walk)
    else:
        np.testing.assert_allclose(scatter[0], walk, rtol=2e-6, atol=1e-7)
    # raw counts (no sample normalisation): the fixed-point unit follows the largest total
    monkeypatch.delenv("UNIFRAC_B200_HYBRID_SCATTER")
    big = ssu_synth.geometric_table(table.obs_ids, 300, 0.02, 5000.0, 66)
    raw_scatter, _ = ssu.one_off_matrix(tree, big, f"{method}_{prec}", normalize=False)
    monkeypatch.setenv("UNIFRAC_B200_HYBRID_SCATTER", "0")
    raw_walk, _ = ssu.one_off_matrix(tree, big, f"{method}_{prec}", normalize=False)
    if prec == "fp64":
        check_fp64(raw_scatter, raw_walk)
    else:
        np.testing.assert_allclose(raw_scatter, raw_walk, rtol=2e-6, atol=1e-4)


@pytest.mark.parametrize("method", ["weighted_normalized", "weighted_unnormalized"])
def test_weighted_fp32_deterministic_mode_repeats_bit_for_bit(ssu, monkeypatch, method):
    """UNIFRAC_B200_DETERMINISTIC=1 gives fp32 plans the owner-per-element
    walk of the sparse rows (no atomics): repeated calls agree bit for bit,
    and with the default (atomic) form to fp32 rounding."""
    tree, table = _case(64, n_tips=400, n_samples=600, density=0.02)
    default, _ = ssu.one_off_matrix(tree, table, f"{method}_fp32")
    monkeypatch.setenv("UNIFRAC_B200_DETERMINISTIC", "1")
    runs = [ssu.one_off_matrix(tree, table, f"{method}_fp32")[0] for _ in range(3)]
    for r in runs[1:]:
        np.testing.assert_array_equal(r, runs[0])
    np.testing.assert_allclose(runs[0], default, rtol=2e-6, atol=1e-7)


UNION_RUNS = [("generalized", False, 0.5), ("generalized", False, 0.0), ("generalized", False, 1.0),
              ("generalized", False, 0.25), ("unweighted", True, 1.0), ("unweighted_unnormalized", True, 1.0),
              ("weighted_normalized", True, 1.0), ("weighted_unnormalized", True, 1.0),
              ("generalized", True, 0.5), ("generalized", True, 0.25)]


@pytest.mark.parametrize("method,vaw,alpha", UNION_RUNS)
def test_union_and_dense_forms_agree(ssu, oracle_mod, monkeypatch, method, vaw, alpha):
    """Generalized and variance-adjusted fp64 pairs summed over the union of
    the two supports (sparse rows) equal the dense form and the oracle; the
    small table splits the node range (split partials + finalize)."""
    tree, table = _case(63, n_tips=400, n_samples=260, density=0.03)
    kw = dict(variance_adjust=vaw, alpha=alpha)
    plan = ssu.Plan(tree, table, method + "_fp64", **kw)
    assert plan.pair_kernel().startswith("pair_union")
    plan.close()
    union, _ = ssu.one_off_matrix(tree, table, method + "_fp64", **kw)
    monkeypatch.setenv("UNIFRAC_B200_UNION_MODE", "dense")
    plan = ssu.Plan(tree, table, method + "_fp64", **kw)
    assert plan.pair_kernel().startswith("pair_values")
    plan.close()
    dense, _ = ssu.one_off_matrix(tree, table, method + "_fp64", **kw)
    check_fp64(union, dense)
    check_fp64(union, oracle_mod.oracle_one_off(tree, table, method + "_fp64", **kw)["matrix"])


@pytest.mark.parametrize("n_tips", [5, 9, 40, 301])
def test_union_rows_stream_in_whole_and_partial_stages(ssu, oracle_mod, n_tips):
    """The union kernel streams the embedded rows 16 at a time: trees whose
    row count is below one stage or not a multiple of 16 (the last stage
    partly past the rows, read as zero) give the oracle's matrix; stripe
    windows go through the same kernel."""
    tree, table = _case(64, n_tips=n_tips, n_samples=150, density=0.3 if n_tips < 40 else 0.05, drop=1)
    kw = dict(variance_adjust=True, alpha=0.5)
    plan = ssu.Plan(tree, table, "generalized_fp64", **kw)
    assert plan.pair_kernel().startswith("pair_union")
    plan.close()
    ref = oracle_mod.oracle_one_off(tree, table, "generalized_fp64", **kw)["matrix"]
    gpu, _ = ssu.one_off_matrix(tree, table, "generalized_fp64", **kw)
    check_fp64(gpu, ref)
    stripes, _ = ssu.partial(tree, table, "generalized_fp64", 10, 40, **kw)
    check_fp64(stripes, oracle_mod.oracle_one_off(tree, table, "generalized_fp64", stripe_start=10, stripe_stop=40,
                                                  **kw)["stripes"])


@pytest.mark.parametrize("method,vaw", [("generalized", False), ("generalized", True), ("weighted_normalized", True),
                                        ("unweighted", True)])
def test_union_fp32_within_reference_fp32_error(ssu, oracle_mod, method, vaw):
    """fp32 inputs through the union kernel (terms in fp64, fp32 output)."""
    tree, table = _case(65, n_tips=400, n_samples=200, density=0.03)
    kw = dict(variance_adjust=vaw, alpha=0.5)
    plan = ssu.Plan(tree, table, method + "_fp32", **kw)
    assert plan.pair_kernel().startswith("pair_union")
    plan.close()
    gpu, _ = ssu.one_off_matrix(tree, table, method + "_fp32", **kw)
    assert gpu.dtype == np.float32
    check_fp32(gpu, oracle_mod, tree, table, method, **kw)


@pytest.mark.parametrize("method", ["unweighted", "weighted_normalized", "weighted_unnormalized", "generalized"])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_negative_counts_take_the_dense_kernels(ssu, oracle_mod, method, prec):
    """Negative entries (the reference accepts them): presence is u > 0, the
    sparse forms need u >= 0, so weighted and generalized plans run the dense
    kernels; results match the oracle (which matches the reference on this
    input)."""
    tree, base = _case(66, n_tips=120, n_samples=70, density=0.15)
    rng = np.random.default_rng(166)
    data = base.data.copy()
    flip = rng.random(data.size) < 0.05
    data[flip] = -0.5 * data[flip]
    table = ssu_synth.Table(base.obs_ids, base.sample_ids, base.indptr, base.indices, data)
    plan = ssu.Plan(tree, table, f"{method}_{prec}", alpha=1.0)
    kernel = plan.pair_kernel()
    plan.close()
    assert "hybrid" not in kernel and "union" not in kernel and "tc" not in kernel
    gpu, _ = ssu.one_off_matrix(tree, table, f"{method}_{prec}", alpha=1.0)
    if prec == "fp64":
        ref = oracle_mod.oracle_one_off(tree, table, method + "_fp64", alpha=1.0)["matrix"]
        assert np.array_equal(np.isnan(gpu), np.isnan(ref))
        check_fp64(gpu, ref)
    else:
        check_fp32(gpu, oracle_mod, tree, table, method, alpha=1.0)


def test_union_wait_that_runs_out_is_an_error_and_the_device_stays_usable(ssu, oracle_mod, monkeypatch):
    """Failure injection without a fault: with UNIFRAC_B200_TEST_STALL the
    union kernel's producer issues no copy, so every consumer's bounded wait
    (here ~1 ms) runs out; the call returns output_error instead of hanging,
    and the next call in the same process is correct."""
    tree, table = _case(67, n_tips=200, n_samples=80, density=0.05)
    kw = dict(variance_adjust=True, alpha=0.5)
    monkeypatch.setenv("UNIFRAC_B200_TEST_STALL", "1")
    monkeypatch.setenv("UNIFRAC_B200_WAIT_CYCLES", "2000000")
    plan = ssu.Plan(tree, table, "generalized_fp64", **kw)
    assert plan.pair_kernel().startswith("pair_union")
    plan.close()
    with pytest.raises(ssu.SSUError) as e:
        ssu.one_off_matrix(tree, table, "generalized_fp64", **kw)
    assert e.value.status == 6  # output_error
    monkeypatch.delenv("UNIFRAC_B200_TEST_STALL")
    monkeypatch.delenv("UNIFRAC_B200_WAIT_CYCLES")
    gpu, _ = ssu.one_off_matrix(tree, table, "generalized_fp64", **kw)
    check_fp64(gpu, oracle_mod.oracle_one_off(tree, table, "generalized_fp64", **kw)["matrix"])


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_hybrid_with_every_row_sparse_matches_dense_form(ssu, monkeypatch, prec):
    """UNIFRAC_B200_HYBRID_DIV=1 sends every row, however dense, through the
    sparse-row path: rows with more than 32 present columns in a 128-column
    block take its chunked branch (fp32) or long walks (fp64)."""
    tree, table = _case(68, n_tips=200, n_samples=300, density=0.3)
    monkeypatch.setenv("UNIFRAC_B200_WEIGHTED_MODE", "dense")
    dense, _ = ssu.one_off_matrix(tree, table, f"weighted_normalized_{prec}")
    monkeypatch.delenv("UNIFRAC_B200_WEIGHTED_MODE")
    monkeypatch.setenv("UNIFRAC_B200_HYBRID_DIV", "1")
    plan = ssu.Plan(tree, table, f"weighted_normalized_{prec}")
    assert plan.pair_kernel().startswith("pair_hybrid")
    plan.close()
    sparse, _ = ssu.one_off_matrix(tree, table, f"weighted_normalized_{prec}")
    if prec == "fp64":
        check_fp64(sparse, dense)
    else:
        np.testing.assert_allclose(sparse, dense, rtol=5e-6, atol=1e-7)


def test_page_locked_results_are_recycled(ssu):
    """Full results of 2 MiB or more come from the page-locked pool, and a
    result released through destroy_mat_full_fp64 goes back to it: after many
    large results, large and smaller ones are still page-locked (flag
    0x2000), so no call falls back to registering pageable memory."""
    import ctypes
    L = ssu.lib()
    tree, table = _case(67, n_tips=300, n_samples=700, density=0.05)
    small_tree, small = _case(68, n_tips=300, n_samples=520, density=0.05)
    for t, tb in [(tree, table)] * 4 + [(small_tree, small)] * 2 + [(tree, table)]:
        x = ssu.Inputs(t, tb)
        res = ctypes.POINTER(ssu.MatFull64)()
        st = L.one_off_matrix_inmem_v3(ctypes.byref(x.biom), ctypes.byref(x.tree), b"weighted_normalized_fp64",
                                       False, 1.0, False, True, 1, 0, False, None, ctypes.byref(res))
        assert st == 0
        assert res.contents.flags & 0x2000, "result not page-locked"
        L.destroy_mat_full_fp64(ctypes.byref(res))


# ---- fp64 unweighted in whole numbers (sample lists + presence words)

def _stripe_mode(monkeypatch, call):
    """`call` with the presence-word stripe form over the embedding (the general path)."""
    monkeypatch.setenv("UNIFRAC_B200_UNWEIGHTED_MODE", "stripe")
    try:
        return call()
    finally:
        monkeypatch.delenv("UNIFRAC_B200_UNWEIGHTED_MODE")


@pytest.mark.parametrize("n,n_tips,density", [(1, 40, 0.2), (2, 40, 0.2), (31, 70, 0.2), (33, 1200, 0.01), (129, 300, 0.9),
                                              (640, 2000, 0.02), (1501, 400, 0.02), (2433, 500, 0.01)])
@pytest.mark.parametrize("method", ["unweighted_fp64", "unweighted_unnormalized_fp64"])
def test_whole_number_unweighted_matches_the_stripe_form(ssu, monkeypatch, method, n, n_tips, density):
    """Both tile shapes (32 x 32 and 128 x 64), nodes by lists alone, by words
    alone and by both, explicit zeros and empty samples, a walk in two parts;
    full matrix, window, condensed, bypassed tips."""
    tree, table = _case(500 + n, n_tips=n_tips, n_samples=n, density=density, drop=5)
    rng = np.random.default_rng(n)
    table.data[rng.random(table.data.shape[0]) < 0.1] = 0.0
    table.data[np.isin(table.indices, [n // 2])] = 0.0
    stop = (n + 1) // 2
    calls = [lambda: ssu.one_off_matrix(tree, table, method)[0],
             lambda: ssu.one_off_matrix(tree, table, method, bypass_tips=True)[0],
             lambda: ssu.one_off(tree, table, method)[0],
             lambda: ssu.partial(tree, table, method, stop // 3, stop)[0]]
    for call in calls if n > 1 else calls[:3]:
        got, ref = call(), _stripe_mode(monkeypatch, call)
        np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
        check_fp64(np.nan_to_num(got), np.nan_to_num(ref))


def test_whole_number_unweighted_close_and_identical_samples(ssu, oracle_mod):
    """Samples equal to another one, or differing by one of the shortest tips:
    their tiles are recomputed in the stripe form."""
    tree, table = _case(77, n_tips=900, n_samples=150, density=0.1, drop=0)
    tree.lengths = np.where(tree.lengths > 0, tree.lengths * 10.0 ** np.random.default_rng(3).uniform(-6, 0, tree.lengths.shape), 0.0)
    dense = table.dense()
    lengths = dict(zip(tree.tip_names(), tree.tip_lengths()))
    shortest = np.argsort([lengths[o] for o in table.obs_ids])
    for j in range(0, 60, 2):
        dense[:, j + 1] = dense[:, j]
        if j % 4 == 0:
            dense[shortest[j % 7], j + 1] = 0.0 if dense[shortest[j % 7], j] > 0 else 3.0
    table = ssu_synth.Table.from_dense(dense, table.obs_ids, table.sample_ids)
    for method in ("unweighted_fp64", "unweighted_unnormalized_fp64"):
        gpu, _ = ssu.one_off_matrix(tree, table, method)
        check_fp64(gpu, oracle_mod.oracle_one_off(tree, table, method)["matrix"])


def test_whole_number_unweighted_in_a_batch_and_as_a_graph(ssu, monkeypatch):
    tree = ssu_synth.random_binary_tree(800, 0.1, 5)
    tips = tree.tip_names()
    tables = [ssu_synth.geometric_table(tips[3 * i:700 + 20 * i], n, 0.05, 10.0, 60 + i)
              for i, n in enumerate((5, 64, 200, 33))]

    def run():
        plan = ssu.BatchPlan(tree, tables, "unweighted_fp64")
        plan.execute()
        first = plan.results()
        plan.set_graph(True)
        for _ in range(2):
            plan.execute()
        for a, b in zip(plan.results(), first):
            np.testing.assert_array_equal(a, b)
        plan.close()
        return first
    for got, ref in zip(run(), _stripe_mode(monkeypatch, run)):
        check_fp64(got, ref)


@pytest.mark.parametrize("what", ["negative length", "infinite count", "negative count"])
def test_whole_number_unweighted_leaves_other_inputs_to_the_stripe_form(ssu, monkeypatch, what):
    tree, table = _case(81, n_tips=300, n_samples=70, density=0.1)
    if what == "negative length":
        tree.lengths = tree.lengths.copy()
        tree.lengths[np.flatnonzero(tree.structure)[5]] = -0.01
    else:
        table.data[3] = np.inf if what == "infinite count" else -2.0
    call = lambda: ssu.one_off_matrix(tree, table, "unweighted_fp64")[0]  # noqa: E731
    np.testing.assert_array_equal(call(), _stripe_mode(monkeypatch, call))


# ---- weighted by sample lists (walk from the tips, lists, dense rows)

def _dense_mode(monkeypatch, call):
    """`call` with the dense pair kernel over the embedding (the general path)."""
    monkeypatch.setenv("UNIFRAC_B200_WEIGHTED_MODE", "dense")
    try:
        return call()
    finally:
        monkeypatch.delenv("UNIFRAC_B200_WEIGHTED_MODE")


def _polytomy(tree, rng):
    """The tree with about a third of its internal nodes merged into their parents."""
    keep = np.ones(len(tree.structure), dtype=bool)
    stack = []
    for i, o in enumerate(tree.structure):
        if o:
            stack.append(i)
        else:
            j = stack.pop()
            if stack and i - j > 1 and rng.random() < 0.35:
                keep[i] = keep[j] = False
    return ssu_synth.BPTree(tree.structure[keep], tree.lengths[keep], [n for n, k in zip(tree.names, keep) if k])


def _check_weighted(got, ref, fp64):
    """fp64: the parity bars.  fp32: the dense fp32 form's own error (sums of
    single-precision terms over every node), as in the comparisons of the sparse
    and dense forms above; 1e-6 of the largest value where two samples are close."""
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    if fp64:
        check_fp64(np.nan_to_num(got), np.nan_to_num(ref))
    else:
        np.testing.assert_allclose(got, ref, rtol=5e-6, atol=1e-6 * max(1.0, float(np.nanmax(np.abs(ref), initial=0))))


@pytest.mark.parametrize("n,n_tips,density", [(1, 40, 0.2), (2, 40, 0.2), (33, 1200, 0.01), (37, 3500, 0.9), (129, 300, 0.9),
                                              (640, 2000, 0.02), (1250, 500, 0.02)])
@pytest.mark.parametrize("method", ["weighted_normalized", "weighted_unnormalized"])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_weighted_by_lists_matches_the_dense_form(ssu, monkeypatch, method, prec, n, n_tips, density):
    """Nodes by lists alone, by rows alone and by both; samples of more nodes
    than shared memory holds (3,500 tips at 90%), a walk in two parts, polytomies,
    explicit zeros and empty samples; full matrix, bypassed tips, raw counts,
    condensed, window."""
    rng = np.random.default_rng(n)
    tree, table = _case(700 + n, n_tips=n_tips, n_samples=n, density=density, drop=5)
    tree = _polytomy(tree, rng)
    table.data[rng.random(table.data.shape[0]) < 0.1] = 0.0
    table.data[np.isin(table.indices, [n // 2])] = 0.0
    m = f"{method}_{prec}"
    stop = (n + 1) // 2
    calls = [lambda: ssu.one_off_matrix(tree, table, m)[0], lambda: ssu.one_off_matrix(tree, table, m, bypass_tips=True)[0],
             lambda: ssu.one_off_matrix(tree, table, m, normalize=False)[0], lambda: ssu.one_off(tree, table, m)[0],
             lambda: ssu.partial(tree, table, m, stop // 3, stop)[0]]
    for call in calls if n > 1 else calls[:4]:
        _check_weighted(call(), _dense_mode(monkeypatch, call), prec == "fp64")


def test_weighted_by_lists_in_a_batch_as_a_graph_and_in_groups(ssu, monkeypatch):
    tree = ssu_synth.random_binary_tree(800, 0.1, 5)
    tips = tree.tip_names()
    tables = [ssu_synth.geometric_table(tips[3 * i:700 + 20 * i], n, 0.05, 10.0, 60 + i)
              for i, n in enumerate((5, 64, 200, 33))]
    for method, fp64 in (("weighted_normalized_fp64", True), ("weighted_unnormalized", False)):
        def run(group_bytes=0, graph=True):
            plan = ssu.BatchPlan(tree, tables, method, group_bytes=group_bytes, autotune=0)
            groups = plan.n_groups()
            plan.execute()
            first = plan.results()
            plan.set_graph(graph)
            for _ in range(2):
                plan.execute()
            for a, b in zip(plan.results(), first):
                np.testing.assert_array_equal(a, b)
            plan.close()
            return first, groups
        (whole, _), (split, groups) = run(), run(group_bytes=1)
        assert groups > 1
        ref, _ = _dense_mode(monkeypatch, run)
        for a, b, c in zip(whole, split, ref):
            _check_weighted(a, c, fp64)
            _check_weighted(b, c, fp64)


@pytest.mark.parametrize("what", ["negative length", "infinite count", "two tips of one name"])
def test_weighted_by_lists_leaves_other_inputs_to_the_embedding(ssu, monkeypatch, what):
    tree, table = _case(83, n_tips=300, n_samples=70, density=0.1)
    if what == "negative length":
        tree.lengths = tree.lengths.copy()
        tree.lengths[np.flatnonzero(tree.structure)[5]] = -0.01
    elif what == "infinite count":
        table.data[3] = np.inf
    else:
        names = [i for i, x in enumerate(tree.names) if x]
        tree.names = list(tree.names)
        tree.names[names[-1]] = tree.names[names[0]]  # (the last tip is not in the table)
    for method in ("weighted_normalized_fp64", "unweighted_fp64"):
        call = lambda: ssu.one_off_matrix(tree, table, method)[0]  # noqa: E731
        ref = _dense_mode(monkeypatch, call) if method.startswith("weighted") else _stripe_mode(monkeypatch, call)
        got = call()
        np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
        check_fp64(np.nan_to_num(got), np.nan_to_num(ref))


# ---- generalized by sample lists (the nodes that both samples have)

def _union_dense(monkeypatch, call):
    """`call` with the dense pair kernel over the embedding (the general path)."""
    monkeypatch.setenv("UNIFRAC_B200_UNION_MODE", "dense")
    try:
        return call()
    finally:
        monkeypatch.delenv("UNIFRAC_B200_UNION_MODE")


@pytest.mark.parametrize("alpha", [0.0, 0.25, 0.5, 1.0, 2.0])
@pytest.mark.parametrize("n,n_tips,density", [(1, 40, 0.2), (2, 40, 0.2), (33, 1200, 0.01), (65, 700, 0.6), (300, 900, 0.03),
                                              (1220, 150, 0.05)])
def test_generalized_by_lists_matches_the_dense_form(ssu, monkeypatch, alpha, n, n_tips, density):
    """Every alpha kind, both tile shapes, nodes by lists, by rows and by both,
    a walk in two parts, polytomies, explicit zeros: full matrix, bypassed tips,
    condensed, window; raw counts stay on the other kernels."""
    rng = np.random.default_rng(n)
    tree, table = _case(900 + n, n_tips=n_tips, n_samples=n, density=density, drop=5)
    tree = _polytomy(tree, rng)
    table.data[rng.random(table.data.shape[0]) < 0.1] = 0.0
    # a table with a sample whose entries are all explicit zeros (0 / 0) stays on
    # the embedding's union kernel: NaN, or where both samples are few items the
    # sparse form's 1, the dense form's NaN
    total = np.bincount(table.indices, weights=table.data, minlength=n)
    void = (total == 0) & (np.bincount(table.indices, minlength=n) > 0)
    k, l = np.triu_indices(n, 1)
    stop = (n + 1) // 2
    s = np.arange(stop // 3, max(stop, stop // 3 + 1))[:, None]
    j = np.arange(n)[None, :]
    m = "generalized_fp64"
    full = void[:, None] | void[None, :]
    calls = [(full, lambda: ssu.one_off_matrix(tree, table, m, alpha=alpha)[0]),
             (full, lambda: ssu.one_off_matrix(tree, table, m, alpha=alpha, bypass_tips=True)[0]),
             (full & False, lambda: ssu.one_off_matrix(tree, table, m, alpha=alpha, normalize=False)[0]),
             (void[k] | void[l], lambda: ssu.one_off(tree, table, m, alpha=alpha)[0]),
             (void[j + 0 * s] | void[(j + s + 1) % n], lambda: ssu.partial(tree, table, m, stop // 3, stop, alpha=alpha)[0])]
    for skip, call in calls if n > 1 else calls[:4]:
        got, ref = call(), _union_dense(monkeypatch, call)
        got, ref = np.where(skip, 0.0, got), np.where(skip, 0.0, ref)
        np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
        check_fp64(np.nan_to_num(got), np.nan_to_num(ref))
    if void.any():
        others = calls[0][1]()[void][:, total > 0]
        assert np.all(np.isnan(others) | (others == 1.0))


@pytest.mark.parametrize("alpha", [0.0, 0.25, 0.5, 2.0])
def test_generalized_by_lists_close_pairs(ssu, oracle_mod, alpha):
    """Near-duplicate samples (their tiles' marked pairs are summed again) meet 1e-12."""
    tree, table = _near_duplicates(62)
    for method in ("generalized_fp64", "generalized"):
        gpu, _ = ssu.one_off_matrix(tree, table, method, alpha=alpha)
        ref = oracle_mod.oracle_one_off(tree, table, "generalized_fp64", alpha=alpha)["matrix"]
        if method.endswith("fp64"):
            check_fp64(gpu, ref)
        else:  # fp64 terms and sums, rounded to single precision once
            np.testing.assert_allclose(gpu, ref, rtol=2.0 ** -23, atol=1e-30)


def test_generalized_by_lists_with_tiny_proportions(ssu, oracle_mod):
    """Proportions down to 1e-30: the branch-free reciprocal square root and the
    lists' fixed point against the oracle."""
    tree, table = _case(91, n_tips=200, n_samples=40, density=0.2)
    rng = np.random.default_rng(4)
    table.data = 10.0 ** rng.uniform(-30, 6, size=table.data.shape)
    for alpha in (0.0, 0.5, 2.0):
        gpu, _ = ssu.one_off_matrix(tree, table, "generalized_fp64", alpha=alpha)
        check_fp64(gpu, oracle_mod.oracle_one_off(tree, table, "generalized_fp64", alpha=alpha)["matrix"])


def test_generalized_by_lists_in_a_batch_as_a_graph(ssu, monkeypatch):
    tree = ssu_synth.random_binary_tree(800, 0.1, 5)
    tips = tree.tip_names()
    tables = [ssu_synth.geometric_table(tips[3 * i:700 + 20 * i], n, 0.05, 10.0, 60 + i)
              for i, n in enumerate((5, 64, 200, 33))]

    def run(group_bytes=0):
        plan = ssu.BatchPlan(tree, tables, "generalized_fp64", alpha=0.5, group_bytes=group_bytes, autotune=0)
        plan.execute()
        first = plan.results()
        plan.set_graph(True)
        for _ in range(2):
            plan.execute()
        for a, b in zip(plan.results(), first):
            np.testing.assert_array_equal(a, b)
        plan.close()
        return first
    for a, b, c in zip(run(), run(group_bytes=1), _union_dense(monkeypatch, run)):
        check_fp64(a, c)
        check_fp64(b, c)


# ---- Faith PD by the walk

@pytest.mark.parametrize("n,n_tips,density", [(1, 3, 1.0), (2, 17, 0.5), (33, 150, 0.3), (70, 400, 0.01), (257, 16, 0.9)])
def test_faith_by_the_walk(ssu, oracle_mod, n, n_tips, density):
    """Bitmaps of one word to many, samples of all tips and of none (explicit
    zeros), chains and polytomies, tips without a table row."""
    rng = np.random.default_rng(n)
    tree, table = _case(700 + n, n_tips=n_tips, n_samples=n, density=density, drop=n_tips // 8)
    tree = _polytomy(tree, rng)
    table.data[rng.random(table.data.shape[0]) < 0.1] = 0.0
    vals, ids = ssu.faith_pd(tree, table)
    ref = oracle_mod.oracle_faith_pd(tree, table)
    np.testing.assert_allclose(vals, ref["values"], rtol=1e-12)


@pytest.mark.parametrize("what", ["negative length", "negative count", "two tips of one name"])
def test_faith_leaves_other_inputs_to_the_embedding(ssu, oracle_mod, what):
    tree, table = _case(84, n_tips=120, n_samples=30, density=0.2)
    if what == "negative length":
        tree.lengths = tree.lengths.copy()
        tree.lengths[np.flatnonzero(tree.structure)[5]] = -0.01
    elif what == "negative count":
        table.data[3] = -0.25 * table.data[3]
    else:
        names = [i for i, x in enumerate(tree.names) if x]
        tree.names = list(tree.names)
        tree.names[names[-1]] = tree.names[names[0]]  # (the last tip is not in the table)
    vals, _ = ssu.faith_pd(tree, table)
    ref = oracle_mod.oracle_faith_pd(tree, table)
    np.testing.assert_allclose(vals, ref["values"], rtol=1e-12)


@pytest.mark.parametrize("method", ["unweighted_fp64", "unweighted", "weighted_normalized_fp64", "weighted_unnormalized",
                                    "generalized_fp64"])
def test_plans_refused_the_lists_memory_are_built_without(ssu, oracle_mod, monkeypatch, method):
    """One table and a batch: the embedding's forms (every node contracted) take over."""
    tree, table = _case(88, n_tips=300, n_samples=150, density=0.1)
    ref = oracle_mod.oracle_one_off(tree, table, method.replace("_fp64", "") + "_fp64", alpha=0.5)["matrix"]
    monkeypatch.setenv("UNIFRAC_B200_TEST_LIST_MEMORY", "1")
    monkeypatch.setenv("UNIFRAC_B200_TC_LISTS", "1")
    plan = ssu.BatchPlan(tree, [table, table], method, alpha=0.5, autotune=0)
    plan.execute()
    for got in [ssu.one_off_matrix(tree, table, method, alpha=0.5)[0], *plan.results()]:
        if method.endswith("fp64"):
            check_fp64(got, ref)
        else:
            np.testing.assert_allclose(got, ref, rtol=1e-6, atol=1e-6)
    plan.close()


# ---- fp32 methods whose results leave as doubles

CRAWFORD = [os.path.join(ROOT, "tests", "golden", "fixtures", f) for f in ("crawford.biom", "crawford.tre")]


@pytest.mark.parametrize("method", ["unweighted", "unweighted_unnormalized", "weighted_normalized", "weighted_unnormalized",
                                    "generalized"])
def test_doubles_of_fp32_methods_keep_the_form_without_lists(ssu, monkeypatch, method):
    """Condensed, stripes, a pair and a file's matrix of an fp32 method are the
    embedding's values bit for bit (as with the lists refused), also where a
    plan of the same table sums its nodes by lists."""
    tree, table = _case(89, n_tips=300, n_samples=150, density=0.1)
    monkeypatch.setenv("UNIFRAC_B200_TC_LISTS", "1")
    monkeypatch.setenv("UNIFRAC_B200_DETERMINISTIC", "1")
    dense = table.dense()
    calls = [lambda: ssu.one_off(tree, table, method, alpha=0.5)[0],
             lambda: ssu.partial(tree, table, method, 10, 40, alpha=0.5)[0],
             lambda: ssu.dense_pair(tree, table.obs_ids, dense[:, 0], dense[:, 1], method, alpha=0.5),
             lambda: ssu.file_matrix("one_off_matrix_v3", *CRAWFORD, method, alpha=0.5)[0]]
    got = [call() for call in calls]
    monkeypatch.setenv("UNIFRAC_B200_TEST_LIST_MEMORY", "1")
    for a, call in zip(got, calls):
        np.testing.assert_array_equal(a, call())


# ---- tables of common features

def _prevalent(seed, n, n_tips, kind):
    """Features that most samples have: prevalences Beta(2, 2) or Beta(5, 2),
    95% of them at 95% and a few at 5%, or all at 90%; every sample has a count."""
    tree = ssu_synth.random_binary_tree(n_tips, 0.1, seed)
    rng = np.random.default_rng(seed)
    p = {"beta22": lambda: rng.beta(2, 2, n_tips), "beta52": lambda: rng.beta(5, 2, n_tips),
         "few rare": lambda: np.where(rng.random(n_tips) < 0.05, 0.05, 0.95), "common": lambda: np.full(n_tips, 0.9)}[kind]()
    dense = np.where(rng.random((n_tips, n)) < p[:, None], rng.geometric(0.1, (n_tips, n)), 0).astype(float)
    dense[rng.integers(n_tips), :] = 2.0
    return tree, ssu_synth.Table.from_dense(dense, tree.tip_names(), ["S%d" % j for j in range(n)])


@pytest.mark.parametrize("kind", ["beta22", "beta52", "few rare"])
@pytest.mark.parametrize("n", [129, 640, 1000, 2048])
def test_whole_number_unweighted_of_common_features(ssu, monkeypatch, kind, n):
    """Nearly all length in dense nodes, a few sparse ones: the fixed point's
    scale follows what a sample sums.  Full matrix, condensed, window, batch."""
    tree, table = _prevalent(n, n, 300, kind)
    stop = (n + 1) // 2

    def batch():
        plan = ssu.BatchPlan(tree, [table, table], "unweighted_fp64", autotune=0)
        plan.execute()
        got = plan.results()[1]
        plan.close()
        return got
    for method in ("unweighted_fp64", "unweighted_unnormalized_fp64"):
        calls = [lambda: ssu.one_off_matrix(tree, table, method)[0], lambda: ssu.one_off(tree, table, method)[0],
                 lambda: ssu.partial(tree, table, method, stop // 3, stop // 3 + 20)[0], batch]
        for call in calls if n == 640 else calls[:1]:
            check_fp64(call(), _stripe_mode(monkeypatch, call))


def test_whole_number_unweighted_with_one_long_stem(ssu, oracle_mod):
    """A small clade under a stem of a thousand times the other lengths, which
    every sample has; the rest of the tree is rare."""
    tree, table = _case(93, n_tips=200, n_samples=300, density=0.05, drop=0)
    inner = [i for i in range(1, len(tree.structure) - 1) if tree.structure[i] and tree.structure[i + 1]]
    dense = table.dense()
    first = table.obs_ids.index(next(nm for nm in tree.names[inner[0]:] if nm))
    dense[first, :] = 1.0
    tree.lengths = tree.lengths.copy()
    tree.lengths[inner[0]] = 1000.0 * tree.lengths.max()
    table = ssu_synth.Table.from_dense(dense, table.obs_ids, table.sample_ids)
    for method in ("unweighted_fp64", "unweighted_unnormalized_fp64"):
        gpu, _ = ssu.one_off_matrix(tree, table, method)
        check_fp64(gpu, oracle_mod.oracle_one_off(tree, table, method)["matrix"])


@pytest.mark.parametrize("alpha", [0.0, 0.5, 1.0, 1.5, 2.0])
@pytest.mark.parametrize("n", [20, 300])
def test_generalized_with_one_long_stem(ssu, oracle_mod, alpha, n):
    """Three quarters of the tree's length (95 of 127) in a stem that every
    sample has whole, so that s^alpha = 2^alpha on it, over eight tips of length
    4 of which a sample has one or two: the denominator is 2.2 (alpha 1.5) and
    3.1 (alpha 2) times the tree's length, and few pairs are close.  (Two more
    tips beside the stem are not in the table.)"""
    structure, lengths, names = [True, True], [0.0, 95.0], ["", ""]
    for i in range(10):
        if i == 8:
            structure.append(False), lengths.append(0.0), names.append("")
        structure += [True, False]
        lengths += [4.0, 0.0]
        names += ["T%d" % i, ""]
    structure.append(False), lengths.append(0.0), names.append("")
    tree = ssu_synth.BPTree(np.array(structure), np.array(lengths), names)
    rng = np.random.default_rng(n)
    dense = np.zeros((8, n))
    for j in range(n):
        dense[rng.integers(8, size=rng.integers(1, 3)), j] = rng.integers(1, 9)
    table = ssu_synth.Table.from_dense(dense, ["T%d" % i for i in range(8)], ["S%d" % j for j in range(n)])
    gpu, _ = ssu.one_off_matrix(tree, table, "generalized_fp64", alpha=alpha)
    check_fp64(gpu, oracle_mod.oracle_one_off(tree, table, "generalized_fp64", alpha=alpha)["matrix"])


@pytest.mark.parametrize("method", ["unweighted_fp64", "weighted_normalized_fp64"])
def test_without_sparse_nodes_the_walk_is_one_launch(ssu, method):
    """2,500 samples that have nearly every tip: the walk, the pair kernel (and
    its split sums), the flagged tiles or close pairs, however many parts a
    list would have."""
    tree, table = _prevalent(7, 2500, 120, "common")
    plan = ssu.Plan(tree, table, method)
    plan.execute()
    plan.result()
    assert plan.launches() <= 4
    plan.close()


# ---- tables of near duplicates (every pair is summed again over its own nodes)

def _all_near(seed, n, n_tips, density):
    """One community with a percent of noise in its counts and a feature or two gained or lost."""
    tree = ssu_synth.random_binary_tree(n_tips, 0.1, seed)
    rng = np.random.default_rng(seed)
    base = rng.random(n_tips) < density
    base[0] = True
    on = base[:, None] ^ (rng.random((n_tips, n)) < 1.0 / n_tips)
    on[0] = True
    counts = np.exp(2 + 1.5 * rng.standard_normal(n_tips))[:, None] * np.exp(0.01 * rng.standard_normal((n_tips, n)))
    dense = np.where(on, np.round(50 * counts) + 1, 0.0)
    return tree, ssu_synth.Table.from_dense(dense, tree.tip_names(), ["S%d" % j for j in range(n)])


@pytest.mark.parametrize("n,n_tips,density", [(2, 30, 0.9), (17, 60, 0.5), (129, 300, 0.2), (150, 9000, 0.002), (300, 700, 0.9)])
@pytest.mark.parametrize("method,alpha", [("weighted_normalized_fp64", 1.0), ("weighted_unnormalized_fp64", 1.0),
                                          ("generalized_fp64", 0.0), ("generalized_fp64", 0.5), ("generalized_fp64", 1.5)])
def test_near_duplicates_are_summed_over_their_own_nodes(ssu, oracle_mod, method, alpha, n, n_tips, density):
    """Strips with every row and column involved and with few, the last ones
    short; samples of fewer and of more nodes than are laid out at once, long
    runs of nodes that none has; full matrix, window, condensed."""
    tree, table = _all_near(n, n, n_tips, density)
    if n == 129:  # half of the samples are like no other
        dense = table.dense()
        rng = np.random.default_rng(5)
        dense[:, ::2] = np.where(rng.random(dense[:, ::2].shape) < 0.3, rng.geometric(0.1, dense[:, ::2].shape), 0.0)
        dense[0] = 4.0
        table = ssu_synth.Table.from_dense(dense, table.obs_ids, table.sample_ids)
    kw = {"alpha": alpha}
    ref = oracle_mod.oracle_one_off(tree, table, method, **kw)["matrix"]
    check_fp64(ssu.one_off_matrix(tree, table, method, **kw)[0], ref)
    if n > 2:
        check_fp64(ssu.one_off(tree, table, method, **kw)[0], ref[np.triu_indices(n, 1)])
        stop = (n + 1) // 2
        s, k = np.arange(stop // 3, stop)[:, None], np.arange(n)[None, :]
        check_fp64(ssu.partial(tree, table, method, stop // 3, stop, **kw)[0], ref[k, (k + s + 1) % n])


@pytest.mark.parametrize("method", ["weighted_normalized_fp64", "generalized_fp64"])
def test_a_table_of_near_duplicates_costs_little_more_than_another(ssu, method):
    """500 samples, every pair close, against 500 unrelated ones with as many
    features: less than eight times as long (a thread a pair took over 60 times)."""
    near = _all_near(11, 500, 4000, 0.05)
    other = _case(11, n_tips=4000, n_samples=500, density=0.05, drop=0)
    best = []
    for tree, table in (near, other):
        plan = ssu.Plan(tree, table, method, alpha=0.5)
        plan.set_timing(True)
        ms = []
        for _ in range(5):
            plan.execute()
            plan.result()
            ms.append(sum(plan.stage_ms()))
        best.append(min(ms))
        plan.close()
    assert best[0] < 8 * best[1], best


# ---- digits of the list sums

def _long_double_matrix(tree, table, method, alpha):
    """Weighted and generalized distances with every step in long double."""
    dense = table.dense()
    row = {o: dense[i] for i, o in enumerate(table.obs_ids)}
    counts, lengths, stack = [], [], [[]]
    for i, o in enumerate(tree.structure):  # a node's counts when its parenthesis closes
        if o:
            stack.append([i, np.zeros(dense.shape[1])])
            if not tree.structure[i + 1] and tree.names[i] in row:
                stack[-1][1] = row[tree.names[i]].copy()
        else:
            at, c = stack.pop()
            if len(stack) > 1:
                stack[-1][1] += c
                counts.append(c)
                lengths.append(tree.lengths[at])
    u = np.array(counts, dtype=np.longdouble) / dense.sum(0).astype(np.longdouble)
    L = np.array(lengths, dtype=np.longdouble)
    u, L = u[(u > 0).any(1)], L[(u > 0).any(1)]
    n = dense.shape[1]
    out = np.zeros((n, n), dtype=np.longdouble)
    for k in range(n - 1):
        s, d = u[:, k:k + 1] + u[:, k + 1:], np.abs(u[:, k:k + 1] - u[:, k + 1:])
        if method.startswith("generalized"):
            p = np.where(s > 0, np.where(s > 0, s, 1) ** np.longdouble(alpha), 0) * L[:, None]
            num, den = (p * d / np.where(s > 0, s, 1)).sum(0), p.sum(0)
        else:
            num, den = (d * L[:, None]).sum(0), (s * L[:, None]).sum(0) if "_normalized" in method else np.longdouble(1)
        out[k, k + 1:] = out[k + 1:, k] = num / den
    return out


@pytest.mark.parametrize("method,alpha", [("generalized_fp64", a) for a in (0.0, 0.25, 0.5, 0.75, 0.9, 1.25, 2.0)]
                         + [("weighted_normalized_fp64", 1.0), ("weighted_unnormalized_fp64", 1.0)])
def test_list_sums_keep_the_digits_of_direct_sums(ssu, monkeypatch, method, alpha):
    """2-norm of the error against long double: no larger than that of the
    embedding's form (the lists refused), give or take a rounding of the result."""
    tree, table = _case(96, n_tips=3000, n_samples=40, density=0.3, drop=0)
    ref = _long_double_matrix(tree, table, method, alpha)

    def error():
        got, _ = ssu.one_off_matrix(tree, table, method, alpha=alpha)
        return np.sqrt(((got - ref) ** 2).sum() / (ref ** 2).sum())
    lists = error()
    monkeypatch.setenv("UNIFRAC_B200_TEST_LIST_MEMORY", "1")
    assert lists <= error() + 2.0 ** -53


@pytest.mark.parametrize("method,alpha", [("generalized_fp64", 0.0), ("generalized_fp64", 0.5), ("weighted_normalized_fp64", 1.0)])
def test_list_sums_of_near_duplicates_keep_the_digits_of_direct_sums(ssu, monkeypatch, method, alpha):
    """The same on near duplicates, some pairs below the bound under which they are
    summed again and some above; give or take two roundings of the result."""
    tree, table = _all_near(97, 96, 2000, 0.05)
    ref = _long_double_matrix(tree, table, method, alpha)

    def error():
        got, _ = ssu.one_off_matrix(tree, table, method, alpha=alpha)
        return np.sqrt(((got - ref) ** 2).sum() / (ref ** 2).sum())
    lists = error()
    monkeypatch.setenv("UNIFRAC_B200_TEST_LIST_MEMORY", "1")
    assert lists <= error() + 2.0 ** -52


def test_fp32_rows_keep_the_digits_of_the_embedding(ssu, monkeypatch):
    """Single precision, samples of 10 to a million reads: the error against long
    double is no larger than that of the embedding's form."""
    tree = ssu_synth.random_binary_tree(2000, 0.1, 98)
    rng = np.random.default_rng(98)
    dense = np.exp(2 + 1.5 * rng.standard_normal((2000, 96))) * 10 ** rng.uniform(0, 4, 96)
    dense = np.where(rng.random(dense.shape) < 0.03, np.round(dense) + 1, 0.0)
    dense[0] += 1.0
    table = ssu_synth.Table.from_dense(dense, tree.tip_names(), ["S%d" % j for j in range(96)])
    ref = _long_double_matrix(tree, table, "weighted_unnormalized", 1.0)
    monkeypatch.setenv("UNIFRAC_B200_DETERMINISTIC", "1")

    def error():
        got = ssu.one_off_matrix(tree, table, "weighted_unnormalized")[0].astype(np.longdouble)
        return np.sqrt(((got - ref) ** 2).sum() / (ref ** 2).sum())
    lists = error()
    monkeypatch.setenv("UNIFRAC_B200_TEST_LIST_MEMORY", "1")
    assert lists <= error()


# ---- lengths and counts far below the largest, and sums out of range

@pytest.mark.parametrize("scale", [1e-6, 1e-11, 1e-30])
@pytest.mark.parametrize("method,alpha", [("unweighted_fp64", 1.0), ("unweighted_unnormalized_fp64", 1.0),
                                          ("weighted_normalized_fp64", 1.0), ("weighted_unnormalized_fp64", 1.0),
                                          ("generalized_fp64", 0.0), ("generalized_fp64", 0.5), ("generalized_fp64", 1.5)])
def test_samples_in_a_clade_of_short_branches(ssu, oracle_mod, method, alpha, scale):
    """Every third sample has only tips of a clade whose branches are 1e-6 to 1e-30
    of the others': few or no units of the fixed point that the table's largest sample sets."""
    tree, table = _case(99, n_tips=300, n_samples=70, density=0.3, drop=0)
    # the first child of the root, its parenthesis and the tips inside
    depth, end = 0, 1
    for end in range(1, len(tree.structure)):
        depth += 1 if tree.structure[end] else -1
        if depth == 0:
            break
    tree.lengths = tree.lengths.copy()
    tree.lengths[1:end] *= scale
    inside = np.array([1 < tree.names.index(o) < end for o in table.obs_ids])
    dense = table.dense()
    dense[np.ix_(~inside, np.arange(70) % 3 == 0)] = 0.0
    dense[np.flatnonzero(inside)[0]] += 2.0
    table = ssu_synth.Table.from_dense(dense, table.obs_ids, table.sample_ids)
    got = ssu.one_off_matrix(tree, table, method, alpha=alpha)[0]
    ref = oracle_mod.oracle_one_off(tree, table, method, alpha=alpha)["matrix"]
    assert np.all(np.isfinite(ref))
    off = np.abs(got - ref) / np.where(ref == 0, 1.0, ref)
    assert off.max() <= FP64_REL, off.max()


@pytest.mark.parametrize("method", ["unweighted_fp64", "weighted_unnormalized_fp64"])
def test_sums_out_of_range_stay_on_the_embedding(ssu, monkeypatch, method):
    """Lengths of 1e306 whose sum is not finite, raw counts: as with the lists refused."""
    tree, table = _case(100, n_tips=300, n_samples=40, density=0.2)
    tree.lengths = np.where(tree.lengths > 0, 1e306, 0.0)
    call = lambda: ssu.one_off_matrix(tree, table, method, normalize=False)[0]  # noqa: E731
    got = call()
    monkeypatch.setenv("UNIFRAC_B200_TEST_LIST_MEMORY", "1")
    np.testing.assert_array_equal(got, call())


@pytest.mark.parametrize("alpha", [0.0, 0.5, 1.0, 1.5])
def test_fp32_generalized_keeps_the_digits_of_the_union_form(ssu, monkeypatch, alpha):
    """Single precision: the error against long double is no larger than the union
    kernel's over the embedding, whose sums are fp64 (alpha 1 too)."""
    tree, table = _case(101, n_tips=1500, n_samples=60, density=0.05, drop=0)
    ref = _long_double_matrix(tree, table, "generalized", alpha)

    def error():
        got = ssu.one_off_matrix(tree, table, "generalized", alpha=alpha)[0].astype(np.longdouble)
        return np.sqrt(((got - ref) ** 2).sum() / (ref ** 2).sum())
    lists = error()
    monkeypatch.setenv("UNIFRAC_B200_TEST_LIST_MEMORY", "1")
    assert lists <= error()


def _duplicates(seed, n, n_tips, density, copies=2):
    """Samples in random order, each with a duplicate (`copies` 1: none) that lacks one of its features half of the time."""
    tree = ssu_synth.random_binary_tree(n_tips, 0.1, seed)
    rng = np.random.default_rng(seed)
    dense = np.where(rng.random((n_tips, n // copies)) < density, rng.geometric(0.1, (n_tips, n // copies)), 0).astype(float)
    dense[0] = 1.0
    dense = np.tile(dense, (1, copies))
    for j in range(n // 2, n, 2):
        dense[rng.choice(np.flatnonzero(dense[1:, j])) + 1, j] = 0.0
    dense = dense[:, rng.permutation(n)]
    return tree, ssu_synth.Table.from_dense(dense, tree.tip_names(), ["S%d" % j for j in range(n)])


@pytest.mark.parametrize("n,n_tips", [(40, 300), (150, 900), (700, 2500)])
def test_whole_number_unweighted_of_duplicated_samples(ssu, monkeypatch, n, n_tips):
    tree, table = _duplicates(n, n, n_tips, 0.05)
    for method in ("unweighted_fp64", "unweighted_unnormalized_fp64"):
        call = lambda: ssu.one_off_matrix(tree, table, method)[0]  # noqa: E731
        check_fp64(call(), _stripe_mode(monkeypatch, call))


def test_duplicated_samples_cost_little_more_than_others(ssu):
    """600 samples, each with a duplicate, against 600 different ones: less than
    twice as long (with every tile of a duplicate in the stripe form over ten times)."""
    best = []
    for copies in (2, 1):
        tree, table = _duplicates(12, 600, 6000, 0.03, copies)
        plan = ssu.Plan(tree, table, "unweighted_fp64")
        plan.set_timing(True)
        ms = []
        for _ in range(5):
            plan.execute()
            plan.result()
            ms.append(sum(plan.stage_ms()))
        best.append(min(ms))
        plan.close()
    assert best[0] < 2 * best[1], best


def test_near_duplicates_of_uneven_depth(ssu, monkeypatch):
    """Raw counts, near duplicates whose depths span a factor of 10,000: the shallow
    pairs are few units of the deepest sample's fixed point, and meet 1e-12 of the dense form."""
    for seed in range(6):
        tree, table = _all_near(200 + seed, 14, 3000, 0.1)
        depth = np.repeat(10.0 ** np.random.default_rng(seed).uniform(0, 4, 7), 2)
        dense = table.dense() * depth
        table = ssu_synth.Table.from_dense(dense, table.obs_ids, table.sample_ids)
        for method in ("weighted_unnormalized_fp64", "weighted_normalized_fp64"):
            call = lambda: ssu.one_off_matrix(tree, table, method, normalize=False)[0]  # noqa: E731
            check_fp64(call(), _dense_mode(monkeypatch, call))
