"""Performance cases of 2pcf_b200: the calls a survey analysis makes, at the
sizes it makes them.

A case is a dict of plain values.  ``prepare`` builds what the calling program
holds before the call (catalogues as float32 CUDA tensors, binning, patch
labels), ``run`` makes one pass through the package's public entry points with
the default context, and ``exact`` restates the result in FP64 with plain
torch where that is affordable.

Results are returned as the reference's own result record holds them
(src/tpcf.f90:17-22: single-precision mean_theta, g_t, g_x, weights, integer
n_pairs); sums per patch and covariances derived from them are stored in the
same single precision, as the reference stores its errors.

Kinds and what they stand for:

  shear       tangential shear around a scalar field, one catalogue pair
              (shear_2pcf): planar or on the sky, with or without a redshift
              cut and a multiplicative bias, per-patch sums for error bars,
              per-lens marks for later re-weighting, log or other binnings
  kappa       scalar-scalar correlation of a map with a field (kappa_2pcf)
  tomography  all (lens bin, source bin) pairs of a survey in one call with the
              block bootstrap and its joint covariance (batch_shear_2pcf,
              block_bootstrap)
  gradient    field-level inference: xi and the gradient of a chi^2 with
              respect to the fields and weights (xi_shear, forward + backward)
  reweight    xi of many foreground maps from stored marks
              (calculate_tpcf_from_marks)
  points      point bootstrap of stored marks (marks_bootstrap)
  patches     k-means patches of a footprint for the block bootstrap
              (partition_data)
"""
import importlib
import math

import numpy as np
import torch

tpcf = importlib.import_module("2pcf_b200")
autograd = importlib.import_module("2pcf_b200.autograd")

ARCMIN = math.pi / 180.0 / 60.0
SKY_LON, SKY_LAT = math.radians(40.0), math.radians(-30.0)
BLOB_SIGMA = 18.0      # arcmin
BLOB_AREA = 3600.0     # one blob per square degree
LENS_SHARE = (0.1, 0.2, 0.4, 0.7, 1.0)     # objects of the tomographic bins,
SOURCE_SHARE = (0.2, 0.5, 1.0, 1.9, 4.0)   # in millions at n_unit = 1e6

SHEAR = dict(kind="shear", spacing="log", clustered=True, zcut=False, bias=False, n_patch=0, marks=False, sky=False)


def listed():
    return [
        # smallest ordinary call: one quick-look measurement on a small field, launches and set-up
        dict(SHEAR, name="shear_20k", n_lens=20_000, n_src=20_000, box=600.0, x_min=1.0, x_max=100.0, n_bin=15,
             clustered=False),
        # small pointed field with a few linear bins, odd sizes
        dict(SHEAR, name="shear_linear_bins", n_lens=30_011, n_src=120_007, box=300.0, x_min=2.0, x_max=60.0,
             n_bin=10, spacing="lin"),
        # one survey field with 100 bootstrap patches
        dict(SHEAR, name="shear_field_2M", n_lens=500_000, n_src=2_000_000, box=1200.0, x_min=1.0, x_max=200.0,
             n_bin=20, n_patch=100),
        # photometric redshifts: sources in front of a lens are cut, shear calibration per source
        dict(SHEAR, name="shear_zcut_bias", n_lens=100_003, n_src=500_009, box=900.0, x_min=1.0, x_max=150.0,
             n_bin=20, zcut=True, bias=True),
        # marks of every lens, stored for later foreground maps
        dict(SHEAR, name="shear_marks", n_lens=100_000, n_src=500_000, box=600.0, x_min=1.0, x_max=100.0, n_bin=20,
             marks=True),
        # the same measurement in sky coordinates
        dict(SHEAR, name="shear_sky", n_lens=100_000, n_src=500_000, box=1200.0, x_min=1.0, x_max=200.0, n_bin=20,
             sky=True),
        # auto-correlation of a convergence map
        dict(kind="kappa", name="kappa_auto_1M", n_lens=1_000_000, box=600.0, x_min=0.5, x_max=250.0, n_bin=30),
        # the whole survey: 10 million objects in 5 x 5 tomographic bins with errors (the largest call)
        dict(kind="tomography", name="tomography_10M", n_unit=1_000_000, box=1897.4, x_min=1.0, x_max=300.0,
             n_bin=20, n_patch=100, n_boot=1000),
        # one gradient step of a field-level fit
        dict(kind="gradient", name="gradient_300k", n_lens=60_000, n_src=300_000, box=600.0, x_min=1.0, x_max=100.0,
             n_bin=15),
        # 16 foreground realisations against stored marks
        dict(kind="reweight", name="reweight_16_maps", n_lens=1_000_000, n_bin=20, n_map=16, n_field=1),
        # error bars of one foreground map by resampling lenses
        dict(kind="points", name="point_bootstrap", n_lens=250_000, n_bin=20, n_boot=1000),
        # bootstrap patches of a survey footprint
        dict(kind="patches", name="patches_1M", n=1_000_000, box=1897.4, k=100),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1


def draw(rng):
    """One more case of the same ranges: survey calls most often, odd sizes."""
    kind = rng.choice(["shear"] * 6 + ["kappa"] * 2 + ["tomography"] * 2 + ["gradient"] * 2 +
                      ["reweight", "points", "patches"])
    if kind == "reweight":
        return dict(kind=kind, n_lens=_log_int(rng, 20_000, 1_500_000), n_bin=rng.randint(8, 40),
                    n_map=rng.randint(1, 40), n_field=rng.randint(1, 4))
    if kind == "points":
        return dict(kind=kind, n_lens=_log_int(rng, 5_000, 500_000), n_bin=rng.randint(8, 32),
                    n_boot=rng.randint(100, 1000))
    if kind == "patches":
        return dict(kind=kind, n=_log_int(rng, 20_000, 2_000_000), box=rng.uniform(300.0, 1900.0),
                    k=rng.randint(20, 200))
    while True:
        box = rng.uniform(300.0, 1900.0)
        x_max = rng.uniform(0.08, 0.4) * box
        c = dict(kind=kind, box=box, x_min=x_max / rng.uniform(30.0, 500.0), x_max=x_max, n_bin=rng.randint(8, 30))
        if kind == "shear":
            c = dict(SHEAR, **c)
            c.update(n_lens=_log_int(rng, 5_000, 1_000_000), n_src=_log_int(rng, 10_000, 4_000_000),
                     spacing=rng.choice(["log"] * 6 + ["lin", "sqrt"]), clustered=rng.random() < 0.7,
                     zcut=rng.random() < 0.25, bias=rng.random() < 0.3, sky=rng.random() < 0.2,
                     n_patch=rng.choice([0, 0, rng.randint(10, 200)]))
            c["marks"] = c["n_lens"] < 400_000 and rng.random() < 0.25
        elif kind == "kappa":
            c.update(n_lens=_log_int(rng, 10_000, 1_000_000))
        elif kind == "tomography":
            c.update(n_unit=_log_int(rng, 10_000, 500_000), n_patch=rng.randint(20, 150),
                     n_boot=rng.randint(100, 1000))
        else:
            c.update(n_lens=_log_int(rng, 5_000, 300_000), n_src=_log_int(rng, 10_000, 1_000_000))
        if _pairs(c) < (1.5e11 if kind == "shear" and c["spacing"] != "log" else 3e11):
            return c


# ------------------------------------------------------------------ inputs --
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, n, lo=0.0, hi=1.0):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _normal(g, n, sigma=1.0):
    return torch.randn(n, generator=g, device="cuda", dtype=torch.float64) * sigma


def _sky_field(g, n_grid=512, slope=-1.5, sigma=0.02):
    """A Gaussian convergence field and its shear (gamma1, gamma2) on a grid."""
    white = torch.fft.fft2(torch.randn(n_grid, n_grid, generator=g, device="cuda", dtype=torch.float64))
    k = torch.fft.fftfreq(n_grid, device="cuda", dtype=torch.float64)
    ky, kx = torch.meshgrid(k, k, indexing="ij")
    k2 = kx * kx + ky * ky
    k2[0, 0] = 1.0
    f = white * k2 ** (slope / 4.0)
    f[0, 0] = 0.0
    kappa = torch.fft.ifft2(f).real
    f = f * (sigma / kappa.std())
    gamma = torch.fft.ifft2(f * torch.complex(kx * kx - ky * ky, 2.0 * kx * ky) / k2)
    return kappa * (sigma / kappa.std()), gamma.real.contiguous(), gamma.imag.contiguous()


def _sample(grid, box, x, y):
    n = grid.shape[0]
    ix = (x / box * n).long().clamp_(0, n - 1)
    iy = (y / box * n).long().clamp_(0, n - 1)
    return grid[iy, ix]


def _positions(g, n, box, clustered):
    """Uniform, or half the objects in Gaussian blobs (galaxy clustering)."""
    x, y = _uniform(g, n, 0.0, box), _uniform(g, n, 0.0, box)
    if clustered:
        m, blobs = n // 2, max(1, int(round(box * box / BLOB_AREA)))
        cx, cy = _uniform(g, blobs, 0.0, box), _uniform(g, blobs, 0.0, box)
        which = torch.randint(0, blobs, (m,), generator=g, device="cuda")
        x[:m] = torch.remainder(cx[which] + _normal(g, m, BLOB_SIGMA), box)
        y[:m] = torch.remainder(cy[which] + _normal(g, m, BLOB_SIGMA), box)
    return x.float(), y.float()


def _lenses(g, n, box, clustered, field, zcut=False):
    x, y = _positions(g, n, box, clustered)
    return dict(x=x, y=y, val=_sample(field[0], box, x, y).float(), w=_uniform(g, n, 0.5, 1.5).float(),
                z=_uniform(g, n, 0.1, 0.7).float() if zcut else torch.zeros(n, device="cuda"))


def _sources(g, n, box, clustered, field, zcut=False, bias=False):
    x, y = _positions(g, n, box, clustered)
    return dict(x=x, y=y, e1=(_sample(field[1], box, x, y) + _normal(g, n, 0.26)).float(),
                e2=(_sample(field[2], box, x, y) + _normal(g, n, 0.26)).float(), w=_uniform(g, n, 0.5, 1.5).float(),
                z=_uniform(g, n, 0.2, 1.2).float() if zcut else torch.ones(n, device="cuda"),
                m=_normal(g, n, 0.02).float() if bias else torch.zeros(n, device="cuda"))


def _to_sky(cat, box):
    lat = SKY_LAT + (cat["y"].double() - box / 2) * ARCMIN
    lon = SKY_LON + (cat["x"].double() - box / 2) * ARCMIN / torch.cos(lat)
    cat["x"], cat["y"] = lon.float(), lat.float()


def _patch_labels(x, y, box, n_patch):
    """Patches in hand: strips x cells of a footprint, n_patch of them."""
    rows = max(1, int(math.sqrt(n_patch)))
    per = [n_patch // rows + (1 if r < n_patch % rows else 0) for r in range(rows)]
    first = torch.tensor(np.concatenate([[0], np.cumsum(per)[:-1]]), device="cuda")
    per = torch.tensor(per, device="cuda")
    r = (y.double() / box * rows).long().clamp_(0, rows - 1)
    c = torch.minimum((x.double() / box * per[r]).long().clamp_(min=0), per[r] - 1)
    return (first[r] + c).int()


def _shear_inputs(case, seed):
    g = _gen(seed)
    field = _sky_field(g)
    box, clustered = case["box"], case.get("clustered", True)
    L = _lenses(g, case["n_lens"], box, clustered, field, case.get("zcut", False))
    S = _sources(g, case["n_src"], box, clustered, field, case.get("zcut", False), case.get("bias", False))
    labels = _patch_labels(L["x"], L["y"], box, case["n_patch"]) if case.get("n_patch", 0) > 0 else None
    if case.get("sky", False):
        _to_sky(L, box)
        _to_sky(S, box)
    return L, S, labels


def _kappa_inputs(case, seed):
    g = _gen(seed)
    kappa = _sky_field(g)[0]
    x, y = _positions(g, case["n_lens"], case["box"], False)
    val, w = _sample(kappa, case["box"], x, y).float(), _uniform(g, case["n_lens"], 0.5, 1.5).float()
    return dict(x=x, y=y, val=val, w=w, kappa_B=_normal(g, case["n_lens"], 0.002).float())


def _marks_inputs(case, seed):
    g = _gen(seed)
    n, nb = case["n_lens"], case["n_bin"]
    n_field = case.get("n_field", 1)
    ns = [n // n_field + (1 if i < n % n_field else 0) for i in range(n_field)]
    fields, val, w = [], [], []
    for m in ns:
        r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
        u = lambda *s: torch.rand(*s, generator=g, device="cuda") + 0.5  # noqa: E731
        fields.append(dict(x=r(m), y=r(m), w=u(m), xi_E=r(m, nb) + 0.1, xi_B=r(m, nb), K=u(m, nb)))
        if case["kind"] == "reweight":
            val.append(0.02 * r(case["n_map"], m) + 0.01)
            w.append(u(case["n_map"], m))
    return fields, val, w


def _unit(case):
    return ARCMIN if case.get("sky", False) else 1.0


def _bins(case):
    return tpcf.create_bins(case["x_min"] * _unit(case), case["x_max"] * _unit(case), case["n_bin"],
                            case.get("spacing", "log"))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "shear":
        L, S, labels = _shear_inputs(case, seed)
        return dict(case=case, bins=_bins(case), labels=labels,
                    field=tpcf.LensingSurveyField(tpcf.LensCatalog(**L), tpcf.ShapeCatalog(**S)))
    if kind == "kappa":
        c = _kappa_inputs(case, seed)
        lenses = tpcf.LensCatalog(x=c["x"], y=c["y"], val=c["val"], w=c["w"])
        kmap = tpcf.KappaMap(x=c["x"], y=c["y"], kappa_E=c["val"], kappa_B=c["kappa_B"], w=c["w"])
        return dict(case=case, bins=_bins(case), field=tpcf.LensingSurveyField(lenses, convergence=kmap))
    if kind == "tomography":
        g = _gen(seed)
        field = _sky_field(g)
        n, box = case["n_unit"], case["box"]
        lenses = [tpcf.LensCatalog(**_lenses(g, int(f * n), box, True, field)) for f in LENS_SHARE]
        shapes = [tpcf.ShapeCatalog(**_sources(g, int(f * n), box, True, field)) for f in SOURCE_SHARE]
        return dict(case=case, bins=_bins(case), lenses=lenses, shapes=shapes, seed=int(seed),
                    labels=[_patch_labels(L.x, L.y, box, case["n_patch"]) for L in lenses],
                    tasks=[(i, j) for i in range(len(lenses)) for j in range(len(shapes))])
    if kind == "gradient":
        L, S, _ = _shear_inputs(case, seed)
        leaves = [t.requires_grad_() for t in (L["val"], L["w"], S["e1"], S["e2"], S["w"])]
        geo = dict(x_A=L["x"], y_A=L["y"], z_A=L["z"], x_B=S["x"], y_B=S["y"], z_B=S["z"], m_B=S["m"])
        return dict(case=case, bins=_bins(case), leaves=leaves, geometry=geo)
    if kind in ("reweight", "points"):
        fields, val, w = _marks_inputs(case, seed)
        return dict(case=case, marks=[tpcf.MarksField(**f) for f in fields], val=val, w=w, seed=int(seed))
    x, y = _positions(_gen(seed), case["n"], case["box"], True)
    return dict(case=case, x=x, y=y, w=torch.ones(case["n"], device="cuda"))


# -------------------------------------------------------------------- pass --
RECORD = ("mean_theta", "g_t", "g_x", "weights", "n_pairs")
MARKS = ("xi_E_marks", "xi_B_marks", "K_marks", "w_marks", "marks_weight")


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "shear":
        r = tpcf.shear_2pcf(state["field"], state["bins"], spherical_coords=case["sky"],
                            calculate_marks=case["marks"], patch_A=state["labels"], n_patch=case["n_patch"])
        out = {k: getattr(r, k) for k in RECORD}
        if case["marks"]:
            out.update({k: getattr(r, k) for k in MARKS})
        if case["n_patch"]:
            out["patch_sums"] = r.patch_sums.astype(np.float32)
        return out
    if kind == "kappa":
        r = tpcf.kappa_2pcf(state["field"], state["bins"], calculate_marks=False)
        return {k: getattr(r, k) for k in RECORD}
    if kind == "tomography":
        rs = tpcf.batch_shear_2pcf(state["lenses"], state["shapes"], state["tasks"], state["bins"],
                                   lens_patches=state["labels"], n_patch=case["n_patch"])
        ps = np.stack([r.patch_sums for r in rs])
        boot = tpcf.block_bootstrap(ps, case["n_boot"], seed=state["seed"])
        out = {k: np.stack([getattr(r, k) for r in rs]) for k in RECORD}
        out.update(patch_sums=ps.astype(np.float32), cov_g_t=boot["cov_g_t"].astype(np.float32),
                   cov_g_x=boot["cov_g_x"].astype(np.float32), multiplicity=boot["multiplicity"])
        return out
    if kind == "gradient":
        xi_t, xi_x = autograd.xi_shear(*state["leaves"], state["geometry"], state["bins"])
        chi2 = (xi_t / GRAD_SIGMA).square().sum() + (xi_x / GRAD_SIGMA).square().sum()
        grads = torch.autograd.grad(chi2, state["leaves"])
        return dict(chi2=chi2.detach().float(), xi_t=xi_t.detach().float(), xi_x=xi_x.detach().float(),
                    **dict(zip(LEAVES, grads)))
    if kind == "reweight":
        return tpcf.calculate_tpcf_from_marks(state["marks"], state["val"], state["w"])
    if kind == "points":
        return tpcf.marks_bootstrap(state["marks"], case["n_boot"], seed=state["seed"])
    labels, centroids, n_iter = tpcf.partition_data(state["x"], state["y"], state["w"], case["k"])
    return dict(labels=labels, centroids=centroids, iterations=n_iter)


GRAD_SIGMA = 1.0e-4
LEAVES = ("d_val_A", "d_w_A", "d_e1_B", "d_e2_B", "d_w_B")


# -------------------------------------------------------------------- work --
def _share(x, box):
    """Probability that two uniform points of a square are closer than x."""
    r = min(x / box, 1.0)
    return math.pi * r * r - 8.0 / 3.0 * r ** 3 + 0.5 * r ** 4


def _pairs(case):
    p = _share(case["x_max"], case["box"]) - _share(case["x_min"], case["box"])
    if case["kind"] == "tomography":
        return sum(LENS_SHARE) * sum(SOURCE_SHARE) * case["n_unit"] ** 2 * p
    if case["kind"] == "kappa":
        return case["n_lens"] ** 2 * p
    return case["n_lens"] * case["n_src"] * p * (0.6 if case.get("zcut", False) else 1.0)


def work(case):
    """Inputs read once, results written once; operations per binned pair:
    26 (shear), 14 (scalar), 52 (shear on the sky), 46 (shear and its
    gradient)."""
    kind = case["kind"]
    if kind in ("reweight", "points"):
        n, nb = case["n_lens"], case["n_bin"]
        m = case["n_map"] if kind == "reweight" else case["n_boot"]
        return dict(bytes=4.0 * n * (3 * nb + 1) + (8.0 * n * m if kind == "reweight" else 0.0),
                    flops=2.0 * n * m * (3 * nb + 1))
    if kind == "patches":  # one assignment pass: six operations per point and centre
        return dict(bytes=16.0 * case["n"], flops=6.0 * case["n"] * case["k"])
    if kind == "tomography":
        byt = (20.0 * sum(LENS_SHARE) + 28.0 * sum(SOURCE_SHARE)) * case["n_unit"]
        return dict(bytes=byt, flops=26.0 * _pairs(case))
    if kind == "kappa":
        return dict(bytes=36.0 * case["n_lens"], flops=14.0 * _pairs(case))
    byt = 20.0 * case["n_lens"] + 28.0 * case["n_src"]
    if kind == "gradient":
        return dict(bytes=byt + 8.0 * case["n_lens"] + 12.0 * case["n_src"], flops=46.0 * _pairs(case))
    if case["marks"]:
        byt += (16.0 * case["n_bin"] + 4.0) * case["n_lens"]
    return dict(bytes=byt, flops=(52.0 if case["sky"] else 26.0) * _pairs(case))


# ------------------------------------------------------------------- exact --
def _edges(case):
    """FP64 bin edges, squared distances or squared chords."""
    lo, hi, n = case["x_min"] * _unit(case), case["x_max"] * _unit(case), case["n_bin"]
    k, spacing = np.arange(n + 1), case.get("spacing", "log")
    if spacing == "log":
        e = 10.0 ** (math.log10(lo) + k * ((math.log10(hi) - math.log10(lo)) / n))
    elif spacing == "lin":
        e = lo + k * ((hi - lo) / n)
    else:
        e = (math.sqrt(lo) + k * ((math.sqrt(hi) - math.sqrt(lo)) / n)) ** 2
    e[0], e[n] = lo, hi
    e2 = (2.0 * np.sin(e / 2.0)) ** 2 if case.get("sky", False) else e * e
    return torch.tensor(e2, device="cuda")


def _vectors(lon, lat):
    return torch.stack([torch.cos(lat) * torch.cos(lon), torch.cos(lat) * torch.sin(lon), torch.sin(lat)])


class _Tiles:
    """All pairs of two catalogues in FP64, tile by tile: lenses in runs of
    similar x against the sources in reach in x."""

    def __init__(self, case, L, S, tile=1 << 22):
        self.sky, self.e2, self.tile = case.get("sky", False), _edges(case), tile
        self.nb, self.zcut = case["n_bin"], case.get("zcut", False)
        reach = case["x_max"] * _unit(case)
        self.key = "y" if self.sky else "x"   # sorted by latitude on the sky
        self.lo = torch.argsort(L[self.key])
        self.so = torch.argsort(S[self.key])
        self.L = {k: v.detach().double()[self.lo] for k, v in L.items()}
        self.S = {k: v.detach().double()[self.so] for k, v in S.items()}
        self.reach = reach * (1.0 + 1e-6)

    def cost(self):
        key = self.key
        span = float(self.S[key].max() - self.S[key].min())
        return self.L[key].numel() * self.S[key].numel() * min(1.0, 2.2 * self.reach / max(span, 1e-30))

    def __iter__(self):
        n, key = self.L[self.key].numel(), self.S[self.key]
        i = 0
        while i < n:
            a = float(self.L[self.key][i]) - self.reach
            s0 = int(torch.searchsorted(key, torch.tensor([a], device="cuda", dtype=torch.float64)))
            guess = int(torch.searchsorted(key, torch.tensor([a + 2.05 * self.reach], device="cuda",
                                                             dtype=torch.float64), right=True)) - s0
            j = min(n, i + max(1, self.tile // max(1, guess)))
            b = float(self.L[self.key][j - 1]) + self.reach
            s1 = int(torch.searchsorted(key, torch.tensor([b], device="cuda", dtype=torch.float64), right=True))
            ls, ss = slice(i, j), slice(s0, s1)
            i = j
            if s1 > s0:
                yield (ls, ss) + self.terms(ls, ss)

    def terms(self, ls, ss):
        """bin (nb = none), distance, cos 2phi, sin 2phi of a tile."""
        L, S = self.L, self.S
        lx, ly, sx, sy = L["x"][ls, None], L["y"][ls, None], S["x"][None, ss], S["y"][None, ss]
        if self.sky:
            ul, us = _vectors(lx, ly), _vectors(sx, sy)
            d = us - ul
            d2 = (d * d).sum(0)
            p = -torch.sin(lx) * d[0] + torch.cos(lx) * d[1]
            q = (-torch.sin(ly) * torch.cos(lx)) * d[0] + (-torch.sin(ly) * torch.sin(lx)) * d[1] + torch.cos(ly) * d[2]
            dist = 2.0 * torch.asin((d2.sqrt() / 2.0).clamp(max=1.0))
        else:
            p, q = lx - sx, ly - sy
            d2 = p * p + q * q
            dist = d2.sqrt()
        b = torch.bucketize(d2, self.e2, right=True) - 1
        b = torch.where(d2 == self.e2[-1], self.nb - 1, b)
        ok = (b >= 0) & (b < self.nb)
        if self.zcut:
            ok &= L["z"][ls, None] <= S["z"][None, ss]
        b = torch.where(ok, b, self.nb)
        s = (p * p + q * q).clamp(min=1e-300)
        return b, dist, (p * p - q * q) / s, 2.0 * p * q / s


def _row_sums(case, L, S, limit):
    """Per lens [n][5][n_bin]: sums of d w, g_t, g_x, w, w (1 + m) over the
    sources of each bin, without the lens's factors; None beyond `limit` pairs."""
    T = _Tiles(case, L, S)
    if T.cost() > limit:
        return None
    nb, SS = T.nb, T.S
    rows = torch.zeros(T.L["x"].numel(), nb, 5, device="cuda", dtype=torch.float64)
    bins = torch.arange(nb, device="cuda")
    for ls, ss, b, dist, c2, s2 in T:
        w = SS["w"][None, ss].expand_as(dist)
        if "e1" in SS:
            e1, e2 = SS["e1"][None, ss], SS["e2"][None, ss]
            t, x = -(e1 * c2 + e2 * s2) * w, (e1 * s2 - e2 * c2) * w
            K = (SS["w"] * (1.0 + SS["m"]))[None, ss].expand_as(dist)
        else:
            t, x = (SS["kappa_E"] * SS["w"])[None, ss].expand_as(dist), (SS["kappa_B"] * SS["w"])[None, ss].expand_as(dist)
            K = w
        hot = (b[:, None, :] == bins[None, :, None]).double()
        rows[ls] += torch.bmm(hot, torch.stack([dist * w, t, x, w, K], dim=2))
    out = torch.zeros_like(rows)
    out[T.lo] = rows
    return out.permute(0, 2, 1)


def _record(rows, val, w):
    val, w = val.detach().double(), w.detach().double()
    dw, t, x, ww, K = (rows[:, q] for q in range(5))
    dw, ww, K = (w[:, None] * dw).sum(0), (w[:, None] * ww).sum(0), (w[:, None] * K).sum(0)
    t, x = ((val * w)[:, None] * t).sum(0), ((val * w)[:, None] * x).sum(0)
    div = lambda a: torch.where(K > 0, a / torch.where(K > 0, K, 1.0), 0.0)  # noqa: E731
    return dict(mean_theta=dw / ww, g_t=div(t), g_x=div(x), weights=ww), (dw, t, x, ww, K)


EXACT_PAIRS = 4.0e10


def exact(case, seed):
    kind = case["kind"]
    if kind == "shear":
        L, S, labels = _shear_inputs(case, seed)
        rows = _row_sums(case, L, S, EXACT_PAIRS)
        if rows is None:
            return None
        out, _ = _record(rows, L["val"], L["w"])
        out["n_pairs"] = None
        if case["marks"]:
            w, vw = L["w"].double()[:, None], (L["val"].double() * L["w"].double())[:, None]
            out.update(xi_E_marks=rows[:, 1] * vw, xi_B_marks=rows[:, 2] * vw, K_marks=rows[:, 4] * w,
                       w_marks=rows[:, 3] * w, marks_weight=(rows[:, 3] * w).sum(1))
        if case["n_patch"]:
            out["patch_sums"] = None
        return out
    if kind == "kappa":
        c = _kappa_inputs(case, seed)
        S = dict(x=c["x"], y=c["y"], kappa_E=c["val"], kappa_B=c["kappa_B"], w=c["w"])
        rows = _row_sums(case, {k: c[k] for k in ("x", "y", "val", "w")}, S, EXACT_PAIRS)
        if rows is None:
            return None
        return dict(_record(rows, c["val"], c["w"])[0], n_pairs=None)
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind == "reweight":
        fields, val, w = _marks_inputs(case, seed)
        per = []
        for f, v, u in zip(fields, val, w):
            u = u.double() * (f["w"].double() * u.double() > 0)
            vu = v.double() * u
            per.append((vu @ f["xi_E"].double(), vu @ f["xi_B"].double(), u @ f["K"].double(), u @ f["w"].double()))
        E, B, K, W = (torch.stack([p[q] for p in per], 1) for q in range(4))
        return dict(g_t=E / K, g_x=B / K, weights=W, g_t_stacked=E.sum(1) / K.sum(1),
                    g_x_stacked=B.sum(1) / K.sum(1), weights_stacked=W.sum(1))
    return None


def _exact_gradient(case, seed):
    L, S, _ = _shear_inputs(case, seed)
    rows = _row_sums(case, L, S, EXACT_PAIRS / 2)
    if rows is None:
        return None
    val, w = L["val"].double(), L["w"].double()
    rec, (_, St, Sx, _, K) = _record(rows, val, w)
    xi_t, xi_x = rec["g_t"], rec["g_x"]
    K = torch.where(K > 0, K, math.inf)
    at, ax = 2.0 * xi_t / GRAD_SIGMA ** 2 / K, 2.0 * xi_x / GRAD_SIGMA ** 2 / K   # d chi2 / d sum g_t, g_x
    ak = -(at * xi_t + ax * xi_x)                                                 # d chi2 / d K
    dv = (rows[:, 1] * at + rows[:, 2] * ax).sum(1)
    out = dict(chi2=(xi_t / GRAD_SIGMA).square().sum() + (xi_x / GRAD_SIGMA).square().sum(), xi_t=xi_t, xi_x=xi_x,
               d_val_A=dv * w, d_w_A=dv * val + (rows[:, 4] * ak).sum(1))
    T = _Tiles(case, L, S)
    pad = lambda a: torch.cat([a, torch.zeros(1, device="cuda", dtype=torch.float64)])  # noqa: E731
    at, ax, ak = pad(at), pad(ax), pad(ak)
    g = torch.zeros(3, T.S["x"].numel(), device="cuda", dtype=torch.float64)
    vw = T.L["val"] * T.L["w"]
    for ls, ss, b, _, c2, s2 in T:
        ct, cx, ck = at[b] * vw[ls, None], ax[b] * vw[ls, None], ak[b] * T.L["w"][ls, None]
        d1, d2 = (-ct * c2 + cx * s2).sum(0), (-ct * s2 - cx * c2).sum(0)   # per unit source weight
        g[0, ss] += d1 * T.S["w"][ss]
        g[1, ss] += d2 * T.S["w"][ss]
        g[2, ss] += d1 * T.S["e1"][ss] + d2 * T.S["e2"][ss] + ck.sum(0) * (1.0 + T.S["m"][ss])
    back = torch.zeros_like(g)
    back[:, T.so] = g
    out.update(d_e1_B=back[0], d_e2_B=back[1], d_w_B=back[2])
    return out
