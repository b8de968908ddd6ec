"""Per-lens outputs, transposed bin chunk by bin chunk on the way out: bin counts
around the chunk (20 bins), lens counts around a block's 32, outputs on the host
and on the device, one patch and several.  The per-lens bars are those of
test_gpu_pairs; counts are exact."""
import numpy as np
import pytest

from conftest import uniform_shear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 19, 20, 21, 45])
@pytest.mark.parametrize("n", [1, 31, 33, 1000])
def test_against_brute_force(tpcf, oracle, ctx, nb, n):
    L, S = uniform_shear(n, 700, 100.0, 300 + nb + n, w="uniform")
    if n > 1:
        L["w"][::9] = 0.0
    bins = tpcf.create_bins(1.0, 60.0, nb)
    res = tpcf.tangential_shear_tpcf(L["x"], L["y"], L["z"], L["val"], L["w"], S["x"], S["y"], S["z"], S["e1"],
                                     S["e2"], S["w"], S["m"], bins, calculate_marks=True, lens_sums=True, ctx=ctx)
    lens = oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq, lens_idx=np.arange(n))["lens"]
    got = res.lens_sums
    np.testing.assert_array_equal(got[:, 5], lens[:, 5])
    # 1e-6 of the lens's sums of term bounds: the terms themselves for the positive
    # quantities, |val| |e| w for the rotated ones
    bound = np.abs(lens)
    bound[:, 1] = bound[:, 2] = np.abs(L["val"])[:, None] * np.hypot(S["e1"], S["e2"]).max() * lens[:, 3]
    assert np.all(np.abs(got[:, :5] - lens[:, :5]) <= 1e-6 * bound[:, :5])
    # the FP32 marks are the FP64 sums rounded once
    for marks, q in ((res.xi_E_marks, 1), (res.xi_B_marks, 2), (res.w_marks, 3), (res.K_marks, 4)):
        np.testing.assert_array_equal(marks, got[:, q].astype(np.float32))
    np.testing.assert_allclose(res.marks_weight, got[:, 3].sum(1), rtol=1.2e-7)


def test_large_host_outputs(tpcf, ctx):
    """More per-lens output than the staging pieces hold at once (64 MiB)."""
    n, nb = 90_000, 20
    L, S = uniform_shear(n, 400, 300.0, 77)
    bins = tpcf.create_bins(1.0, 60.0, nb)
    res = tpcf.tangential_shear_tpcf(L["x"], L["y"], L["z"], L["val"], L["w"], S["x"], S["y"], S["z"], S["e1"],
                                     S["e2"], S["w"], S["m"], bins, calculate_marks=False, lens_sums=True, ctx=ctx)
    assert res.lens_sums.nbytes > 64 << 20
    np.testing.assert_array_equal(res.lens_sums[:, 5].sum(0), res.n_pairs)
    for i in range(0, n, 9973):
        d2 = (np.float64(L["x"][i]) - S["x"]) ** 2 + (np.float64(L["y"][i]) - S["y"]) ** 2
        np.testing.assert_array_equal(res.lens_sums[i, 5], np.histogram(d2, bins.bin_edges_sq)[0])


@pytest.mark.parametrize("sky", [False, True])
def test_workspace_of_a_batch_of_many_tasks(tpcf, sky):
    """60 tasks with per-lens sums: the split groups' extra columns are bounded for the
    call, not only per task (1.7 GB of sums in all, 8 times that with 8 sets each);
    sums per bin as when launched alone, bit for bit, per lens to FP64 rounding."""
    ctx = tpcf.Context(0)
    L, S = uniform_shear(30_000, 2000, 400.0, 350, w="uniform")
    unit = np.pi / 180 / 60 if sky else 1.0
    for c in (L, S):
        c["x"], c["y"] = (c["x"] * unit).astype(np.float32), ((c["y"] - 200.0) * unit).astype(np.float32)
    lens = tpcf.LensCatalog(L["x"], L["y"], L["val"], L["w"], L["z"])
    src = tpcf.ShapeCatalog(*(S[k] for k in ("x", "y", "e1", "e2", "w", "z", "m")))
    bins = tpcf.create_bins(1.0 * unit, 20.0 * unit, 20)
    unsplit = 8 * 6 * 20 * 30_000
    res = tpcf.batch_shear_2pcf([lens], [src], [(0, 0)] * 60, bins, lens_sums="device", spherical_coords=sky, ctx=ctx)
    held = ctx.stats()["workspace_bytes"]
    alone = tpcf.batch_shear_2pcf([lens], [src], [(0, 0)], bins, lens_sums="device", spherical_coords=sky, ctx=ctx)[0]
    ctx.close()
    assert held <= 1.25 * (60 * unsplit + (1 << 30))   # a slot is a quarter larger than asked for
    ref = alone.lens_sums.cpu().numpy()
    for r in res:
        for k in ("n_pairs", "sum_gt", "sum_gx", "sum_w", "sum_dw", "sum_K"):
            np.testing.assert_array_equal(getattr(r, k), getattr(alone, k))
        got = r.lens_sums.cpu().numpy()
        np.testing.assert_array_equal(got[:, 5], ref[:, 5])
        np.testing.assert_allclose(got[:, 3], ref[:, 3], rtol=1e-12)
        np.testing.assert_allclose(got[:, 1], ref[:, 1], rtol=1e-12, atol=1e-12)
    assert abs(alone.lens_sums[:, 3].sum().item() - alone.sum_w.sum()) <= 1e-9 * alone.sum_w.sum()


@pytest.mark.parametrize("n", [13_000, 13_108, 200_000])
def test_large_host_outputs_at_odd_addresses(tpcf, ctx, monkeypatch, n):
    """Marks of around and well above 1 MiB each into host memory that starts and ends
    inside pages: the values of the device-independent sums, and nothing outside."""
    L, S = uniform_shear(n, 3000, 600.0, 360, w="uniform")
    bins = tpcf.create_bins(1.0, 15.0, 20)
    alloc, held = tpcf._alloc_result, []

    def odd(nb, nA, *a):
        r, c = alloc(nb, nA, *a)
        for k in ("xi_E_marks", "xi_B_marks", "K_marks", "w_marks"):
            buf = np.full(nA * nb + 64, 7.0, np.float32)
            held.append(buf)
            r[k] = buf[3:3 + nA * nb].reshape(nA, nb)
            setattr(c, k, r[k].ctypes.data)
        return r, c
    monkeypatch.setattr(tpcf, "_alloc_result", odd)
    res = tpcf.tangential_shear_tpcf(L["x"], L["y"], L["z"], L["val"], L["w"], S["x"], S["y"], S["z"], S["e1"],
                                     S["e2"], S["w"], S["m"], bins, calculate_marks=True, lens_sums=True, ctx=ctx)
    for buf in held:
        assert np.all(buf[:3] == 7.0) and np.all(buf[3 + n * 20:] == 7.0)
    for k, q in (("xi_E_marks", 1), ("xi_B_marks", 2), ("K_marks", 4), ("w_marks", 3)):
        np.testing.assert_array_equal(getattr(res, k), res.lens_sums[:, q].astype(np.float32))
