"""Partial sums of the marks: every tiling of the rows (n_bin decides how many
tiles of 8 the xi and the K rows fill), lens counts around a warp's group of 16,
arrays that do not start on a 16-byte boundary, and both forms (n_bin <= 32 and
wider) over several passes.  FP64 throughout, so the results agree with numpy's
FP64 products to the rounding of the summation order (1e-9 relative to the sums
of |terms|; at most 1e3 lenses)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def on_device(a, skew):
    import torch
    flat = torch.empty(a.size + 1, dtype=torch.float32, device="cuda")
    view = flat[skew:skew + a.size].view(a.shape)
    view.copy_(torch.from_numpy(a))
    return view


@pytest.mark.parametrize("skew", [0, 1])
@pytest.mark.parametrize("nb", [1, 4, 5, 8, 9, 12, 13, 16, 17, 20, 21, 24, 25, 28, 31, 32, 33])
def test_tilings(tpcf, ctx, nb, skew):
    rng = np.random.default_rng(100 * nb + skew)
    for n, n_map in ((1, 1), (15, 9), (16, 16), (66, 17), (1000, 35)):
        f = lambda *s: rng.normal(0.5, 1.0, s).astype(np.float32)
        xE, xB, K = f(n, nb), f(n, nb), rng.uniform(0.5, 1.5, (n, nb)).astype(np.float32)
        mw = np.where(rng.uniform(size=n) < 0.1, -1.0, rng.uniform(0.5, 1.5, n)).astype(np.float32)
        mw[0] = 1.0
        val, w = f(n_map, n), rng.uniform(0.5, 1.5, (n_map, n)).astype(np.float32)
        d = lambda a: on_device(a, skew)
        field = tpcf.MarksField(x=d(f(n)), y=d(f(n)), w=d(mw), xi_E=d(xE), xi_B=d(xB), K=d(K))
        out = tpcf.calculate_tpcf_from_marks([field], [d(val)], [d(w)], ctx=ctx)
        u = w.astype(np.float64) * (mw > 0)   # lenses of no positive weight are dropped
        vu = val.astype(np.float64) * u
        Ks = u @ K.astype(np.float64)
        for key, xi in (("g_t", xE), ("g_x", xB)):
            x64 = xi.astype(np.float64)
            band = 1e-9 * (np.abs(vu) @ np.abs(x64)) / Ks
            assert np.all(np.abs(np.asarray(out[key])[:, 0] - vu @ x64 / Ks) <= band), (n, key)
        np.testing.assert_allclose(np.asarray(out["weights"])[:, 0], u @ mw.astype(np.float64), rtol=1e-12)


@pytest.mark.parametrize("labels", [False, True])
@pytest.mark.parametrize("nb", [7, 40])
def test_draws_of_several_passes(tpcf, oracle, ctx, nb, labels):
    """Several passes drawn and summed per launch: each resample is the one that
    its counter gives, whatever launch it falls in."""
    rng = np.random.default_rng(nb)
    n, n_boot, n_unit = 203, 75, 41
    f = lambda *s: rng.normal(0.5, 1.0, s).astype(np.float32)
    m = tpcf.MarksField(x=f(n), y=f(n), w=rng.uniform(0.5, 1.5, n).astype(np.float32), xi_E=f(n, nb), xi_B=f(n, nb),
                        K=rng.uniform(0.5, 1.5, (n, nb)).astype(np.float32))
    unit = rng.integers(0, n_unit, n).astype(np.int32) if labels else None
    units = n_unit if labels else n
    kw = dict(units=unit, n_units=n_unit) if labels else {}
    out = tpcf.marks_bootstrap([m], n_boot, seed=11, covariance=False, ctx=ctx, **kw)
    mult = oracle.bootstrap_multiplicity(11, n_boot, units, units).astype(np.float64)
    per_lens = mult[:, unit] if labels else mult
    np.testing.assert_allclose(out["weights"], per_lens @ m.w.astype(np.float64), rtol=1e-12)
    K = per_lens @ m.K.astype(np.float64)
    x64 = m.xi_E.astype(np.float64)
    band = 1e-9 * (per_lens @ np.abs(x64)) / K
    assert np.all(np.abs(out["g_t"] - per_lens @ x64 / K) <= band)
