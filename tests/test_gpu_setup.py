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
