"""k-means passes that settle most points by distance bounds: labels, centroids
and pass count equal the plain search of the oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def f32(a):
    return np.ascontiguousarray(a, np.float32)


def points(kind, n, rng):
    if kind == "lattice":        # many exact ties between centroids
        s = int(np.ceil(np.sqrt(n)))
        g = np.stack(np.meshgrid(np.arange(s), np.arange(s)), -1).reshape(-1, 2)[:n]
        return f32(g[:, 0]), f32(g[:, 1])
    if kind == "clumps":         # some starting cells are empty
        c = rng.uniform(0, 500, (5, 2))
        p = c[rng.integers(0, 5, n)] + rng.normal(0, 3, (n, 2))
        return f32(p[:, 0]), f32(p[:, 1])
    if kind == "far":            # a large offset: coordinates carry few digits
        return f32(1e4 + rng.uniform(0, 40, n)), f32(-2e4 + rng.uniform(0, 90, n))
    if kind == "copies":
        p = rng.uniform(0, 100, (max(1, n // 50), 2))[rng.integers(0, max(1, n // 50), n)]
        return f32(p[:, 0]), f32(p[:, 1])
    return f32(rng.uniform(0, 1900, n)), f32(rng.uniform(0, 600, n))


@pytest.mark.parametrize("kind,n,k,zero_w", [("lattice", 4097, 16, False), ("lattice", 900, 25, True),
                                             ("clumps", 3001, 30, False), ("far", 5000, 12, False),
                                             ("copies", 2500, 7, True), ("uniform", 1024, 2, False),
                                             ("uniform", 1023, 40, False), ("uniform", 200_003, 90, False)])
def test_passes_equal_the_plain_search(tpcf, oracle, ctx, kind, n, k, zero_w):
    rng = np.random.default_rng(n + k)
    x, y = points(kind, n, rng)
    w = f32(rng.uniform(0.2, 1.5, n))
    if zero_w:
        w[rng.random(n) < 0.3] = 0.0
    lab, cen, it = tpcf.partition_data(x, y, w, k, ctx=ctx)
    lab_o, cen_o, it_o = oracle.kmeans_det(x, y, w, k)
    assert it == it_o
    np.testing.assert_array_equal(lab, lab_o)
    np.testing.assert_array_equal(cen, cen_o)


@pytest.mark.parametrize("max_iter,tol", [(0, 0.0), (1, 0.0), (7, 0.0), (20, 0.0), (1000, 0.02)])
def test_stopping_rules(tpcf, oracle, ctx, max_iter, tol):
    rng = np.random.default_rng(5)
    x, y = points("uniform", 20_000, rng)
    w = f32(rng.uniform(0.2, 1.5, 20_000))
    lab, cen, it = tpcf.partition_data(x, y, w, 20, iterations=max_iter, reassignment_tol=tol, ctx=ctx)
    lab_o, cen_o, it_o = oracle.kmeans_det(x, y, w, 20, max_iter, tol)
    assert it == it_o
    np.testing.assert_array_equal(lab, lab_o)
    np.testing.assert_array_equal(cen, cen_o)


@pytest.mark.parametrize("n", [3, 63, 64, 65, 18_943, 18_944, 18_945, 606_207, 606_209])
def test_points_of_a_block(tpcf, oracle, ctx, n):
    """Around the steps of the number of points that a block takes at a time."""
    rng = np.random.default_rng(n)
    x, y = points("uniform", n, rng)
    w = f32(rng.uniform(0.2, 1.5, n))
    k = 2 if n < 63 else 11
    lab, cen, it = tpcf.partition_data(x, y, w, k, iterations=12, ctx=ctx)
    lab_o, cen_o, it_o = oracle.kmeans_det(x, y, w, k, 12, 0.0)
    assert it == it_o
    np.testing.assert_array_equal(lab, lab_o)
    np.testing.assert_array_equal(cen, cen_o)
