"""Failure paths, made to happen without a GPU fault or hang
(tpcf_debug_inject; the reference stops the program instead,
src/kdtree.f90:119-122, :265-267):

- a device workspace allocation that fails at one of several points of a
  call returns TPCF_ERR_OOM with its message, and the same context then
  computes the correct result;
- a source tile of the pair kernel whose bulk copy is never issued makes the
  bounded mbarrier waits on it run out: the call returns TPCF_ERR_TIMEOUT
  (every copy that was issued has landed before the blocks exit), and the
  same context then computes the correct result;
- the same for the first tile of the marks kernel (xi from marks and the
  marks bootstrap).
Invalid arguments and a missing device are covered on the CPU (test_abi)."""
import ctypes as C
import time

import numpy as np
import pytest

from conftest import uniform_shear
from parity import check_sums

pytestmark = pytest.mark.gpu


def shear(tpcf, ctx, L, S, bins):
    return tpcf.tangential_shear_tpcf(L["x"], L["y"], L["z"], L["val"], L["w"], S["x"], S["y"], S["z"],
                                      S["e1"], S["e2"], S["w"], S["m"], bins, calculate_marks=False, ctx=ctx)


def inject(tpcf, ctx, fail_alloc=-1, skip_tile=-1, wait_polls=0):
    st = tpcf._lib.lib().tpcf_debug_inject(ctx.handle, int(fail_alloc), int(skip_tile), C.c_uint32(wait_polls))
    assert st == tpcf._lib.TPCF_OK


@pytest.mark.parametrize("k", [0, 4, 12, 30])
def test_injected_allocation_failure_then_recovery(tpcf, oracle, k):
    ctx = tpcf.Context(0)
    L, S = uniform_shear(2000, 3000, 200.0, 80 + k)
    bins = tpcf.create_bins(1.0, 40.0, 10)
    can = oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq)
    if k == 30:
        shear(tpcf, ctx, L, S, bins)   # a warm context: the failing allocation is a regrowth
        S = {q: np.concatenate([v, v]) for q, v in S.items()}
        can = oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq)
    inject(tpcf, ctx, fail_alloc=k if k < 30 else 0)
    with pytest.raises(tpcf.TPCFError) as e:
        shear(tpcf, ctx, L, S, bins)
    assert e.value.status == tpcf._lib.TPCF_ERR_OOM
    assert "allocation" in str(e.value)
    check_sums(f"call after an injected allocation failure at workspace allocation {k}", shear(tpcf, ctx, L, S, bins),
               can)
    ctx.close()


def test_bounded_wait_runs_out_then_recovery(tpcf, oracle):
    ctx = tpcf.Context(0)
    L, S = uniform_shear(3000, 20000, 300.0, 90)
    bins = tpcf.create_bins(1.0, 60.0, 12)
    can = oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq)
    for tile, polls in ((0, 1 << 12), (5, 1 << 16)):
        inject(tpcf, ctx, skip_tile=tile, wait_polls=polls)
        t0 = time.time()
        with pytest.raises(tpcf.TPCFError) as e:
            shear(tpcf, ctx, L, S, bins)
        dt = time.time() - t0
        assert e.value.status == tpcf._lib.TPCF_ERR_TIMEOUT, str(e.value)
        print(f"tile {tile} never issued, {polls} polls per wait: TIMEOUT after {dt:.3f} s")
    inject(tpcf, ctx)
    check_sums("call after a bounded wait ran out", shear(tpcf, ctx, L, S, bins), can)
    ctx.close()


@pytest.mark.parametrize("kind", ["series", "sphere"])
def test_bounded_wait_of_the_series_and_spherical_kernels(tpcf, oracle, kind):
    """The same for the kernel of dense source catalogues and the one on the sky."""
    ctx = tpcf.Context(0)
    L, S = uniform_shear(400, 60_000, 60.0, 91)
    unit = np.pi / 180 / 60 if kind == "sphere" else 1.0
    for c in (L, S):
        c["x"], c["y"] = (c["x"] * unit).astype(np.float32), (c["y"] * unit).astype(np.float32)
    bins = tpcf.create_bins(0.5 * unit, 20.0 * unit, 8)
    kw = dict(calculate_marks=False, spherical_coords=kind == "sphere", ctx=ctx)
    call = lambda: tpcf.tangential_shear_tpcf(L["x"], L["y"], L["z"], L["val"], L["w"], S["x"], S["y"], S["z"],  # noqa: E731
                                              S["e1"], S["e2"], S["w"], S["m"], bins, **kw)
    for tile, polls in ((0, 1 << 12), (4, 1 << 14)):
        inject(tpcf, ctx, skip_tile=tile, wait_polls=polls)
        with pytest.raises(tpcf.TPCFError) as e:
            call()
        assert e.value.status == tpcf._lib.TPCF_ERR_TIMEOUT, str(e.value)
    inject(tpcf, ctx)
    can = (oracle.canon_sphere(oracle.SHEAR, L, S, bins.chord_edges_sq) if kind == "sphere" else
           oracle.canon_pairs(oracle.SHEAR, L, S, bins.bin_edges_sq))
    check_sums(f"{kind} call after a bounded wait ran out", call(), can)
    ctx.close()


def test_marks_bounded_wait_runs_out_then_recovery(tpcf, oracle):
    ctx = tpcf.Context(0)
    rng = np.random.default_rng(92)
    n, nb, n_map = 8192, 20, 3
    raw = {"x": rng.normal(size=n).astype(np.float32), "y": rng.normal(size=n).astype(np.float32),
           "w": rng.uniform(0.1, 2, n).astype(np.float32),
           "xi_E": rng.normal(size=(n, nb)).astype(np.float32), "xi_B": rng.normal(size=(n, nb)).astype(np.float32),
           "K": rng.uniform(0.5, 1.5, (n, nb)).astype(np.float32)}
    marks = [tpcf.MarksField(**raw)]
    val = rng.normal(0, 0.02, (n_map, n)).astype(np.float32)
    w = rng.uniform(0.5, 1.5, (n_map, n)).astype(np.float32)
    inject(tpcf, ctx, skip_tile=0, wait_polls=1 << 12)
    for call in (lambda: tpcf.calculate_tpcf_from_marks(marks, [val], [w], ctx=ctx),
                 lambda: tpcf.marks_bootstrap(marks, 20, seed=3, covariance=False, ctx=ctx)):
        with pytest.raises(tpcf.TPCFError) as e:
            call()
        assert e.value.status == tpcf._lib.TPCF_ERR_TIMEOUT, str(e.value)
    inject(tpcf, ctx)
    out = tpcf.calculate_tpcf_from_marks(marks, [val], [w], ctx=ctx)
    for m in range(n_map):
        per, _ = oracle.xi_from_marks([raw], [val[m]], [w[m]])
        np.testing.assert_allclose(out["g_t"][m, 0], per[0]["g_t"], rtol=1e-9)
        np.testing.assert_allclose(out["weights"][m, 0], per[0]["weights"], rtol=1e-12)
    ctx.close()


HOST_MEMORY = """
import importlib, resource, sys
import numpy as np
sys.path.insert(0, {root!r})
tpcf = importlib.import_module("2pcf_b200")
from importlib import import_module
rng = np.random.default_rng(1)
f = lambda *s: rng.uniform(0.5, 1.0, s).astype(np.float32)
marks = [tpcf.MarksField(x=f(64), y=f(64), w=f(64), xi_E=f(64, 20), xi_B=f(64, 20), K=f(64, 20))]
ctx = tpcf.Context(0)
ref = tpcf.marks_bootstrap(marks, 8, seed=1, covariance=False, ctx=ctx)["g_t"]
held = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (held + (4 << 30), resource.RLIM_INFINITY))
files = import_module("2pcf_b200.files")
arr, keep = files._cfields(marks)
st = tpcf._lib.lib().tpcf_marks_bootstrap(ctx.handle, 1, arr, None, 0, None, 1, 50_000_000, 1.0, 1, None, None, None,
                                          None, None)
assert st == tpcf._lib.TPCF_ERR_OOM, st
again = tpcf.marks_bootstrap(marks, 8, seed=1, covariance=False, ctx=ctx)["g_t"]
assert np.array_equal(ref, again)
print("returned")
"""


def test_host_allocation_failure_is_a_status():
    """Sums that do not fit the process's address space (a limit set for it): the entry
    point returns TPCF_ERR_OOM, and the context stays usable."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", HOST_MEMORY.format(root=root)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "returned" in r.stdout, (r.returncode, r.stderr[-800:])
