"""The series pair kernel (dense source catalogues without per-lens outputs):
sub-chunk moments, direct passes at bin edges, ragged groups and sub-chunks,
against the FP64 oracle.  Bar as in test_gpu_pairs: n_pairs bit-exact, every sum
within 1e-6 of the oracle's sum of |terms| (FP32 pair terms, FP64 sums; the series
is truncated below 1e-7 of a sub-chunk's sum of |terms|)."""
import numpy as np
import pytest

from parity import check_sums

pytestmark = pytest.mark.gpu

N_SRC, BOX = 60_001, 60.0   # sub-chunks of about 1.4' a side, the last one ragged


def f32(a):
    return np.ascontiguousarray(a, np.float32)


def catalogues(seed, n_lens, n_src=N_SRC, z=False):
    rng = np.random.default_rng(seed)
    L = dict(x=f32(rng.uniform(0, BOX, n_lens)), y=f32(rng.uniform(0, BOX, n_lens)),
             z=f32(rng.uniform(0, 0.8, n_lens)) if z else np.zeros(n_lens, np.float32),
             val=f32(rng.normal(0.01, 0.02, n_lens)), w=f32(rng.uniform(0.5, 1.5, n_lens)))
    S = dict(x=f32(rng.uniform(0, BOX, n_src)), y=f32(rng.uniform(0, BOX, n_src)),
             z=f32(rng.uniform(0.1, 1.2, n_src)) if z else np.ones(n_src, np.float32),
             e1=f32(rng.normal(0, .26, n_src)), e2=f32(rng.normal(0, .26, n_src)),
             w=f32(rng.uniform(0.5, 1.5, n_src)), m=f32(rng.normal(0, .03, n_src)) if z else np.zeros(n_src, np.float32))
    return L, S


def shear(tpcf, ctx, L, S, bins, **kw):
    return tpcf.tangential_shear_tpcf(L["x"], L["y"], L["z"], L["val"], L["w"], S["x"], S["y"], S["z"], S["e1"],
                                      S["e2"], S["w"], S["m"], bins, calculate_marks=False, ctx=ctx, **kw)


@pytest.mark.parametrize("n_lens,z", [(1, False), (63, False), (64, True), (65, False), (200, True)])
def test_log_bins(tpcf, oracle, ctx, n_lens, z):
    L, S = catalogues(60 + n_lens, n_lens, z=z)
    bins = tpcf.create_bins(0.3, 25.0, 8)
    res = shear(tpcf, ctx, L, S, bins)
    check_sums(f"series log {n_lens} lenses z={z}", res, oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq))


@pytest.mark.parametrize("spacing,lo", [("lin", 0.0), ("sqrt", 0.5), ("ihs", 0.2)])
def test_other_spacings(tpcf, oracle, ctx, spacing, lo):
    L, S = catalogues(71, 70)
    bins = tpcf.create_bins(lo, 20.0, 12, spacing=spacing, p=0.5)
    res = shear(tpcf, ctx, L, S, bins)
    check_sums(f"series {spacing}", res, oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq))


def test_coincident_pair_in_the_first_linear_bin(tpcf, oracle, ctx):
    """A lens on a source with x_min = 0: the pair counts, its d is 0, its g
    terms are 0/0 in bin 0 and nowhere else."""
    L, S = catalogues(72, 66)
    L["x"][5], L["y"][5] = S["x"][777], S["y"][777]
    bins = tpcf.create_bins(0.0, 20.0, 10, spacing="lin")
    res = shear(tpcf, ctx, L, S, bins)
    can = oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq)
    np.testing.assert_array_equal(res.n_pairs, can["n_pairs"].astype(np.int64))
    assert np.isnan(res.sum_gt[0]) and np.all(np.isfinite(res.sum_gt[1:]))
    assert np.all(np.abs(res.sum_gt[1:] - can["sum_gt"][1:]) <= 1e-6 * can["abs_gt"][1:])
    np.testing.assert_allclose(res.sum_dw, can["sum_dw"], rtol=1e-6)


def test_kappa_auto_correlation(tpcf, oracle, ctx):
    rng = np.random.default_rng(73)
    n = 20_011
    x, y = f32(rng.uniform(0, BOX, n)), f32(rng.uniform(0, BOX, n))
    k, w = f32(rng.normal(0, .02, n)), f32(rng.uniform(0.5, 1.5, n))
    kb = f32(rng.normal(0, .01, n))
    bins = tpcf.create_bins(0.5, 25.0, 5)
    res = tpcf.scalar_kappa_tpcf(x, y, k, w, x, y, k, kb, w, bins, calculate_marks=False, ctx=ctx)
    L = dict(x=x, y=y, val=k, w=w)
    K = dict(x=x, y=y, kappa_E=k, kappa_B=kb, w=w)
    check_sums("series kappa auto", res, oracle.canon_pairs(oracle.KAPPA, L, K, bins.bin_edges_sq))


def test_pairs_on_the_edges(tpcf, oracle, ctx):
    """Dense rings within a few ulp of every edge: decided in FP64."""
    bins = tpcf.create_bins(1.0, 25.0, 6)
    rng = np.random.default_rng(74)
    n = 60_000
    d = bins.bin_edges[rng.integers(0, 7, n)] * (1.0 + rng.integers(-40, 41, n) * 1e-8)
    a = rng.uniform(0, 2 * np.pi, n)
    _, S = catalogues(74, 1, n_src=n)
    S["x"], S["y"] = f32(30 + d * np.cos(a)), f32(30 + d * np.sin(a))
    L = dict(x=np.full(3, 30, np.float32), y=np.full(3, 30, np.float32), z=np.zeros(3, np.float32),
             val=np.ones(3, np.float32), w=np.ones(3, np.float32))
    res = shear(tpcf, ctx, L, S, bins)
    check_sums("series rings", res, oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq))


def test_patches_and_mixed_batch(tpcf, oracle, ctx):
    """A dense and a sparse source catalogue in one batch (two pair kernels):
    each task as when launched alone, patch sums adding up to the totals."""
    rng = np.random.default_rng(75)
    L, S = catalogues(75, 150)
    _, S2 = catalogues(76, 1, n_src=500)
    bins = tpcf.create_bins(0.5, 25.0, 8)
    lab = rng.integers(0, 5, 150).astype(np.int32)
    lc = tpcf.LensCatalog(L["x"], L["y"], L["val"], L["w"], L["z"])
    sc = [tpcf.ShapeCatalog(s["x"], s["y"], s["e1"], s["e2"], s["w"], s["z"], s["m"]) for s in (S, S2)]
    both = tpcf.batch_shear_2pcf([lc], sc, [(0, 0), (0, 1)], bins, lens_patches=[lab], n_patch=5, ctx=ctx)
    for i, s in enumerate((S, S2)):
        check_sums(f"series mixed batch {i}", both[i], oracle.canon_pairs(oracle.SHEAR, L, s, bins.bin_edges_sq))
        one = tpcf.batch_shear_2pcf([lc], [sc[i]], [(0, 0)], bins, lens_patches=[lab], n_patch=5, ctx=ctx)[0]
        np.testing.assert_array_equal(one.patch_sums, both[i].patch_sums)
        np.testing.assert_array_equal(both[i].patch_sums[:, 5].sum(0), both[i].n_pairs)


@pytest.mark.parametrize("n_same", [31, 32, 64])
def test_coincident_sources_fill_a_sub_chunk(tpcf, oracle, ctx, n_same):
    """Sources on one point, the first of the sorted catalogue (its lowest corner), and
    a lens on the same point: with bins from 0 those pairs count, their d is 0 and their
    g terms are 0/0 in bin 0 and nowhere else, also where they fill whole sub-chunks."""
    L, S = catalogues(77, 66)
    S["x"], S["y"] = f32(np.maximum(S["x"], 0.25)), f32(np.maximum(S["y"], 0.25))
    S["x"][:n_same], S["y"][:n_same] = 0.0, 0.0
    L["x"][5], L["y"][5] = 0.0, 0.0
    bins = tpcf.create_bins(0.0, 20.0, 5, spacing="lin")
    res = shear(tpcf, ctx, L, S, bins)
    can = oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq)
    np.testing.assert_array_equal(res.n_pairs, can["n_pairs"].astype(np.int64))
    assert np.isnan(res.sum_gt[0]) and np.isnan(res.sum_gx[0])
    assert np.all(np.abs(res.sum_gt[1:] - can["sum_gt"][1:]) <= 1e-6 * can["abs_gt"][1:])
    assert np.all(np.abs(res.sum_gx[1:] - can["sum_gx"][1:]) <= 1e-6 * can["abs_gx"][1:])
    np.testing.assert_allclose(res.sum_dw, can["sum_dw"], rtol=1e-6)
    np.testing.assert_allclose(res.sum_w, can["sum_w"], rtol=1e-6)


@pytest.mark.parametrize("lens_w,src_w,val", [(1e-25, 1e-25, 1.0), (1e-20, 1e-15, 1e-25), (1e22, 1e25, 1.0),
                                              (1e30, 1e-30, 1e30)])
def test_very_small_and_large_weights(tpcf, oracle, ctx, lens_w, src_w, val):
    """Weights in physical units: lens and source factors that each fit FP32 while
    their product does not."""
    L, S = catalogues(78, 130)
    L["w"], L["val"], S["w"] = f32(L["w"] * lens_w), f32(L["val"] * val), f32(S["w"] * src_w)
    bins = tpcf.create_bins(0.3, 25.0, 8)
    res = shear(tpcf, ctx, L, S, bins)
    check_sums(f"series weights {lens_w} {src_w} {val}", res,
               oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq))


@pytest.mark.parametrize("unit", [1e-13, 1e-16])
@pytest.mark.parametrize("spacing,lo", [("log", 0.3), ("lin", 0.0)])
def test_very_small_coordinates(tpcf, oracle, ctx, spacing, lo, unit):
    """Positions and bins in a unit that makes squared separations tiny (still normal
    FP32 numbers): relative accuracy as at any other scale."""
    L, S = catalogues(79, 130)
    for c in (L, S):
        c["x"], c["y"] = f32(c["x"] * unit), f32(c["y"] * unit)
    bins = tpcf.create_bins(lo * unit, 25.0 * unit, 8, spacing=spacing)
    res = shear(tpcf, ctx, L, S, bins)
    check_sums(f"series unit {unit} {spacing}", res, oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq))


def test_sub_chunks_of_two_knots(tpcf, oracle, ctx):
    """Every sub-chunk two knots of sources with equal values, 31 and 1 of them at its
    two ends, just far enough for the series: all their truncation errors add up.
    Truncation is at most 4.6e-8 (g) and 2e-8 (d) of the terms; FP32 gives 1/d^2 and d
    errors of up to 2.6e-7 and 1.3e-7 (twice and once the 2^-22.9 of a reciprocal
    square root) of either sign at 225 different distances, so their mean stays well
    below half of that: bars of 2.5e-7 of the sum of |e| w and 1.5e-7 of the sum of d w."""
    rng = np.random.default_rng(80)
    gy, gx = np.meshgrid(30.0 + 60.0 * np.arange(15), 30.0 + 60.0 * np.arange(15), indexing="ij")
    gx, gy = gx.ravel(), gy.ravel()
    end = np.where(np.arange(32) < 31, 1.0, -1.0)
    n_fill = 100_000   # away from every lens: the catalogue is dense on average
    x = np.concatenate([(gx[:, None] + end).ravel(), rng.uniform(840, 900, n_fill)])
    y = np.concatenate([np.repeat(gy, 32), rng.uniform(960, 1000, n_fill)])
    n = x.size
    S = dict(x=f32(x), y=f32(y), z=np.ones(n, np.float32), e1=np.full(n, .3, np.float32),
             e2=np.full(n, .1, np.float32), w=np.ones(n, np.float32), m=np.zeros(n, np.float32))
    r, a = rng.uniform(12.55, 12.75, gx.size), np.radians(70.0)
    L = dict(x=f32(gx - r * np.cos(a)), y=f32(gy - r * np.sin(a)), z=np.zeros(gx.size, np.float32),
             val=np.ones(gx.size, np.float32), w=np.ones(gx.size, np.float32))
    bins = tpcf.create_bins(8.0, 20.0, 1, spacing="lin")
    res = shear(tpcf, ctx, L, S, bins)
    can = oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq)
    assert can["n_pairs"][0] == 32 * 225
    check_sums("series knots", res, can)
    d_g = np.hypot(res.sum_gt[0] - can["sum_gt"][0], res.sum_gx[0] - can["sum_gx"][0]) / (32 * 225 * np.hypot(.3, .1))
    d_d = abs(res.sum_dw[0] - can["sum_dw"][0]) / can["sum_dw"][0]
    print("knots:", d_g, d_d)
    assert d_g <= 2.5e-7 and d_d <= 1.5e-7


def test_tasks_of_a_mixed_batch(tpcf, ctx, monkeypatch):
    """Tasks with and without marks, calibration in one source catalogue only, dense and
    sparse sources: each task's sums are those of the task alone, bit for bit (sum_K,
    which a call without calibration copies from sum_w, to the last places of FP64)."""
    rng = np.random.default_rng(81)
    def source(n, m):
        return tpcf.ShapeCatalog(f32(rng.uniform(0, 300, n)), f32(rng.uniform(0, 300, n)), f32(rng.normal(0, .26, n)),
                                 f32(rng.normal(0, .26, n)), f32(rng.uniform(.5, 1.5, n)), np.ones(n, np.float32),
                                 f32(rng.normal(0, .03, n)) if m else np.zeros(n, np.float32))
    n = 300
    lens = tpcf.LensCatalog(f32(rng.uniform(0, 300, n)), f32(rng.uniform(0, 300, n)), f32(rng.normal(0, .02, n)),
                            f32(rng.uniform(.5, 1.5, n)), np.zeros(n, np.float32))
    src = [source(300_000, False), source(30_000, False), source(40_000, True)]
    bins = tpcf.create_bins(1.0, 100.0, 20)
    tasks = [(0, 0, False), (0, 0, True), (0, 1, False), (0, 1, True), (0, 2, False)]
    alloc = tpcf._alloc_result

    def run(sources, what):
        marks = iter([t[2] for t in what])
        monkeypatch.setattr(tpcf, "_alloc_result", lambda nb, nA, _, *a: alloc(nb, nA, next(marks), *a))
        return tpcf.batch_shear_2pcf([lens], sources, [t[:2] for t in what], bins, ctx=ctx)
    together = run(src, tasks)
    for t in range(len(tasks)):
        alone = run([src[tasks[t][1]]], [(0, 0, tasks[t][2])])[0]
        for k in ("n_pairs", "sum_gt", "sum_gx", "sum_w", "sum_dw"):
            np.testing.assert_array_equal(getattr(together[t], k), getattr(alone, k), err_msg=f"task {t} {k}")
        np.testing.assert_allclose(together[t].sum_K, alone.sum_K, rtol=1e-14)
        if tasks[t][2]:
            np.testing.assert_array_equal(together[t].xi_E_marks, alone.xi_E_marks)


@pytest.mark.parametrize("cut,calibration", [(True, False), (False, True), (True, True)])
@pytest.mark.parametrize("spacing,lo", [("log", 0.3), ("lin", 0.0), ("sqrt", 0.5)])
def test_cut_and_calibration_apart(tpcf, oracle, ctx, spacing, lo, cut, calibration):
    L, S = catalogues(82, 97, z=True)
    if not cut:
        L["z"][:] = 0.0
    if not calibration:
        S["m"][:] = 0.0
    bins = tpcf.create_bins(lo, 20.0, 9, spacing=spacing, p=0.5)
    res = shear(tpcf, ctx, L, S, bins)
    check_sums(f"series {spacing} cut={cut} m={calibration}", res,
               oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq))


@pytest.mark.parametrize("spacing,lo", [("lin", 0.0), ("sqrt", 0.5)])
def test_kappa_other_spacings(tpcf, oracle, ctx, spacing, lo):
    """Scalar-scalar, lenses drawn from the sources: d = 0 counts in bin 0 from x_min = 0
    and leaves the sums finite (they hold no angle)."""
    L, S = catalogues(83, 70)
    L["x"][:30], L["y"][:30] = S["x"][:30], S["y"][:30]
    bins = tpcf.create_bins(lo, 20.0, 9, spacing=spacing)
    res = tpcf.scalar_kappa_tpcf(L["x"], L["y"], L["val"], L["w"], S["x"], S["y"], S["e1"], S["e2"], S["w"], bins,
                                 calculate_marks=False, ctx=ctx)
    K = dict(x=S["x"], y=S["y"], kappa_E=S["e1"], kappa_B=S["e2"], w=S["w"])
    check_sums(f"series kappa {spacing}", res, oracle.canon_pairs(oracle.KAPPA, L, K, bins.bin_edges_sq))


def test_values_that_are_not_finite(tpcf, ctx):
    """A NaN ellipticity and an infinite weight reach the bins of their own pairs and no
    others: far away from every lens, none."""
    L, S = catalogues(84, 40)
    L["x"], L["y"] = f32(L["x"] * 0.3), f32(L["y"] * 0.3)
    bins = tpcf.create_bins(0.5, 12.0, 6)
    clean = shear(tpcf, ctx, L, S, bins)
    gone = np.flatnonzero((S["x"] > 45) & (S["y"] > 45))
    S["e1"][gone[0]], S["w"][gone[1]] = np.nan, np.inf
    res = shear(tpcf, ctx, L, S, bins)
    for k in ("n_pairs", "sum_gt", "sum_gx", "sum_w", "sum_dw"):
        np.testing.assert_array_equal(getattr(res, k), getattr(clean, k))
    one = np.argmin(np.hypot(S["x"] - L["x"][0], S["y"] - L["y"][0]))
    S["e1"][one] = np.nan
    res = shear(tpcf, ctx, L, S, bins)
    np.testing.assert_array_equal(res.n_pairs, clean.n_pairs)
    assert np.isnan(res.sum_gt).any() and np.all(np.isfinite(res.sum_w)) and np.all(np.isfinite(res.sum_dw))
