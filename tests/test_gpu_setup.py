"""Set-up of a pair call: sort keys of any width, work items ordered in one block
or by a radix sort, groups of one and of many patches.  The totals must be the
oracle's (bar of test_gpu_pairs) and independent of patches and shards."""
import numpy as np
import pytest

from conftest import uniform_shear
from parity import check_sums

pytestmark = pytest.mark.gpu


def shear(tpcf, ctx, L, S, bins, **kw):
    return tpcf.tangential_shear_tpcf(L["x"], L["y"], L["z"], L["val"], L["w"], S["x"], S["y"], S["z"], S["e1"],
                                      S["e2"], S["w"], S["m"], bins, calculate_marks=False, ctx=ctx, **kw)


@pytest.mark.parametrize("n_patch", [1, 2, 255, 256, 1000, 70_000])
def test_patch_counts(tpcf, oracle, ctx, n_patch):
    """70 000 patches need 64-bit lens keys; most are empty."""
    rng = np.random.default_rng(n_patch)
    L, S = uniform_shear(3000, 2000, 200.0, 91)
    L["w"][::50] = 0.0
    bins = tpcf.create_bins(1.0, 40.0, 6)
    lab = rng.integers(0, n_patch, 3000).astype(np.int32)
    lab[:3] = n_patch - 1
    res = shear(tpcf, ctx, L, S, bins, patch_A=lab, n_patch=n_patch)
    check_sums(f"{n_patch} patches", res, oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq))
    used = np.unique(lab[L["w"] != 0])
    n = res.patch_sums[:, 5].sum(1)
    assert np.all(n[np.setdiff1d(np.arange(n_patch), used)] == 0)
    np.testing.assert_array_equal(res.patch_sums[:, 5].sum(0), res.n_pairs)


@pytest.mark.parametrize("n_lens", [31, 33, 90_000, 600_000])
def test_item_counts(tpcf, ctx, n_lens):
    """2, 16, about 8 000 and 18 750 work items (the last beyond one block's
    sort); shards add up to the whole call."""
    L, S = uniform_shear(n_lens, 300, 300.0, n_lens)
    bins = tpcf.create_bins(1.0, 20.0, 4)
    res = shear(tpcf, ctx, L, S, bins)
    d2 = lambda i: (L["x"][i:i + 4000, None].astype(np.float64) - S["x"]) ** 2 + \
        (L["y"][i:i + 4000, None].astype(np.float64) - S["y"]) ** 2
    n = sum(np.histogram(d2(i), bins.bin_edges_sq)[0] for i in range(0, n_lens, 4000))
    np.testing.assert_array_equal(res.n_pairs, n)
    parts = []
    for r in range(3):
        ctx.set_shard(r, 3)
        parts.append(shear(tpcf, ctx, L, S, bins))
    ctx.set_shard(0, 0)
    np.testing.assert_array_equal(sum(p.n_pairs for p in parts), n)
    np.testing.assert_allclose(sum(p.sum_gt for p in parts), res.sum_gt, rtol=0, atol=1e-12 * np.abs(res.sum_w).max())


def test_contexts_on_several_threads(tpcf):
    """One context per host thread, each with its own bins, clusters and marks (other
    amounts of shared memory for the same kernels): the results of a thread alone."""
    import threading
    rng = np.random.default_rng(91)
    f = lambda a: np.ascontiguousarray(a, np.float32)  # noqa: E731
    L, S = uniform_shear(3000, 20_000, 100.0, 92, w="uniform")
    work = [(8, False, 5), (20, True, 90), (31, True, 400), (60, True, 20)]
    marks = [[tpcf.MarksField(x=f(rng.normal(size=4000)), y=f(rng.normal(size=4000)), w=f(rng.uniform(.5, 1, 4000)),
                              xi_E=f(rng.normal(size=(4000, nb))), xi_B=f(rng.normal(size=(4000, nb))),
                              K=f(rng.uniform(.5, 1, (4000, nb))))] for nb, _, _ in work]

    def calls(ctx, i):
        nb, per_lens, k = work[i]
        r = tpcf.tangential_shear_tpcf(L["x"], L["y"], L["z"], L["val"], L["w"], S["x"], S["y"], S["z"], S["e1"],
                                       S["e2"], S["w"], S["m"], tpcf.create_bins(1.0, 30.0, nb),
                                       calculate_marks=per_lens, ctx=ctx)
        b = tpcf.marks_bootstrap(marks[i], 20, seed=2, covariance=False, ctx=ctx)
        q = tpcf.partition_data(S["x"], S["y"], S["w"], k, iterations=15, ctx=ctx)
        return [r.n_pairs, r.sum_gt, b["g_t"], q[0], q[1]] + ([r.xi_E_marks] if per_lens else [])
    ctx = tpcf.Context(0)
    alone = [calls(ctx, i) for i in range(len(work))]
    ctx.close()
    wrong = []

    def thread(i):
        try:
            c = tpcf.Context(0)
            for _ in range(15):
                for a, b in zip(calls(c, i), alone[i]):
                    np.testing.assert_array_equal(a, b)
            c.close()
        except BaseException as e:  # noqa: BLE001
            wrong.append((i, repr(e)[:300]))
    threads = [threading.Thread(target=thread, args=(i,)) for i in range(len(work))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong, wrong
