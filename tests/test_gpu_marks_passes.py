"""Marks passes: maps and resamples in groups of 16, several passes' partial sums
reduced together, device draws overlapped with the sums.  FP64 throughout, so
the results agree with numpy's FP64 products to the rounding of the summation
order (1e-9 relative to sums of |terms|; up to 2e3 lenses)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def marks(tpcf, rng, n, nb):
    f = lambda *s: rng.normal(0.5, 1.0, s).astype(np.float32)
    return tpcf.MarksField(x=f(n), y=f(n), w=rng.uniform(0.5, 1.5, n).astype(np.float32), xi_E=f(n, nb), xi_B=f(n, nb),
                           K=rng.uniform(0.5, 1.5, (n, nb)).astype(np.float32))


@pytest.mark.parametrize("n_map,nb,ns", [(1, 5, (70,)), (16, 32, (64, 129)), (17, 20, (500, 1, 300)), (40, 8, (1000,))])
def test_maps(tpcf, ctx, n_map, nb, ns):
    rng = np.random.default_rng(n_map)
    F = [marks(tpcf, rng, n, nb) for n in ns]
    val = [rng.normal(0, 1, (n_map, n)).astype(np.float32) for n in ns]
    w = [rng.uniform(0.5, 1.5, (n_map, n)).astype(np.float32) for n in ns]
    out = tpcf.calculate_tpcf_from_marks(F, val, w, ctx=ctx)
    for i, m in enumerate(F):
        vw = val[i].astype(np.float64) * w[i]
        K = w[i].astype(np.float64) @ m.K
        band = 1e-9 * (np.abs(vw) @ np.abs(m.xi_E.astype(np.float64))) / K
        assert np.all(np.abs(out["g_t"][:, i] - vw @ m.xi_E / K) <= band)
        np.testing.assert_allclose(out["weights"][:, i], w[i].astype(np.float64) @ m.w, rtol=1e-12)


@pytest.mark.parametrize("n_boot,nb,n", [(1, 6, 80), (16, 20, 65), (17, 20, 700), (2721, 32, 2048)])
def test_resamples(tpcf, ctx, n_boot, nb, n):
    """The largest case needs two reductions (169 passes kept at most)."""
    rng = np.random.default_rng(n_boot)
    m = marks(tpcf, rng, n, nb)
    mult = rng.poisson(1.0, (n_boot, n)).astype(np.int32)
    out = tpcf.marks_bootstrap([m], n_boot, multiplicity=mult, covariance=False, ctx=ctx)
    M = mult.astype(np.float64)
    K = M @ m.K
    band = 1e-9 * (M @ np.abs(m.xi_E.astype(np.float64))) / K
    assert np.all(np.abs(out["g_t"] - M @ m.xi_E / K) <= band)
    np.testing.assert_allclose(out["weights"], M @ m.w, rtol=1e-12)
    # device draws: n draws per resample, the same every call
    a = tpcf.marks_bootstrap([m], n_boot, seed=3, covariance=False, ctx=ctx)
    b = tpcf.marks_bootstrap([m], n_boot, seed=3, covariance=False, ctx=ctx)
    for k in ("g_t", "g_x", "weights"):
        np.testing.assert_array_equal(a[k], b[k])
    assert np.all(a["weights"] >= n * 0.5) and np.all(a["weights"] <= n * 1.5)
