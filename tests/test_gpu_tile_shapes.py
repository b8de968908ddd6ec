"""The tile shape of a call that sets none follows from the bins and the sums per
bin.  Counts are the oracle's for every shape.  Shapes share the arithmetic of a
pair and differ in the order of the sums only: at most 144 terms are added in
FP32 before FP64 takes over, so two shapes agree to 2 x 144 x 2^-24 = 1.8e-5 of the
sum of |terms| at worst."""
import numpy as np
import pytest

from conftest import uniform_shear
from parity import check_sums

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("calibration", [False, True])
@pytest.mark.parametrize("nb", [17, 20, 21, 23, 26, 30, 35, 40, 60])
def test_shapes(tpcf, oracle, ctx, nb, calibration):
    L, S = uniform_shear(700, 2500, 300.0, nb)
    L["z"][:] = np.random.default_rng(nb).uniform(0, 1, 700)
    S["z"][:] = np.random.default_rng(nb + 1).uniform(0, 1, 2500)
    S["m"][:] = 0.1 * np.cos(np.arange(2500)) if calibration else 0.0
    bins = tpcf.create_bins(1.0, 60.0, nb)
    can = oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq)
    first = None
    for shape in ((0, 0), (128, 2), (128, 1), (64, 2), (32, 2)):
        ctx.set_tile_shape(*shape)
        try:
            res = tpcf.tangential_shear_tpcf(L["x"], L["y"], L["z"], L["val"], L["w"], S["x"], S["y"], S["z"], S["e1"],
                                             S["e2"], S["w"], S["m"], bins, calculate_marks=False, ctx=ctx)
        finally:
            ctx.set_tile_shape(0, 0)
        np.testing.assert_array_equal(res.n_pairs, can["n_pairs"])
        first = res if first is None else first
        for k, scale in (("sum_gt", "abs_gt"), ("sum_gx", "abs_gx"), ("sum_w", "sum_w"), ("sum_K", "sum_K"),
                         ("sum_dw", "sum_dw")):
            assert np.all(np.abs(getattr(res, k) - getattr(first, k)) <= 1.8e-5 * np.abs(can[scale])), (shape, k)


@pytest.mark.parametrize("calibration", [False, True])
@pytest.mark.parametrize("nb", [17, 21, 30, 40])
def test_shapes_against_brute_force(tpcf, oracle, ctx, nb, calibration):
    """Every shape within the bars of test_gpu_pairs, and all of them the same bit for bit:
    neither the terms nor the folds into FP64 depend on the tiles."""
    L, S = uniform_shear(2000, 9000, 300.0, 100 + nb, w="uniform")
    S["m"][:] = 0.1 * np.cos(np.arange(9000)) if calibration else 0.0
    bins = tpcf.create_bins(1.0, 200.0, nb)
    can = oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq)
    first = None
    for shape in ((0, 0), (128, 2), (128, 1), (64, 2), (32, 2)):
        ctx.set_tile_shape(*shape)
        try:
            res = tpcf.tangential_shear_tpcf(L["x"], L["y"], L["z"], L["val"], L["w"], S["x"], S["y"], S["z"], S["e1"],
                                             S["e2"], S["w"], S["m"], bins, calculate_marks=False, ctx=ctx)
        finally:
            ctx.set_tile_shape(0, 0)
        check_sums(f"shape {shape}, {nb} bins", res, can)
        first = res if first is None else first
        for k in ("sum_gt", "sum_gx", "sum_w", "sum_K", "sum_dw"):
            np.testing.assert_array_equal(getattr(res, k), getattr(first, k))
