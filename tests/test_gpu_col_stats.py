"""Per-gene sums in every order of entries (needs a B200).

The statistics kernel joins two 32-entry steps when 64 genes increase, and
falls back to runs of increasing genes otherwise: sorted rows of every length
around the steps, unsorted rows, and one gene repeated through a step, in the
three value types, with one and several passes of genes.  Every product and sum
is FP64, so the sums agree with FP64 sums in another order to 1e-12 of the sum
of magnitudes (a few thousand terms of 1.1e-16).
"""

import ctypes as C

import numpy as np
import pytest

from scx_b200 import _lib

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def _rows(kind, g, rng):
    if kind == "sorted":
        lengths = [0, 1, 31, 32, 33, 63, 64, 65, 0, 127, 128, 129, 255, 256, 257, 500] * 40
        return [np.sort(rng.choice(g, min(m, g), replace=False)) for m in lengths]
    if kind == "unsorted":
        return [rng.integers(0, g, m) for m in rng.integers(0, 200, 300)]
    return [np.full(m, g - 1) for m in (1, 32, 64, 300)]  # one gene, again and again


CASES = [(kind, g, dtype) for kind in ("sorted", "unsorted", "repeated") for g in (1, 40, 700, 2000, 12800)
         for dtype in ("float32", "bfloat16", "float16")]
# several passes of genes: through a plan, which sorts its rows and converts its values
CASES.append(("sorted", 13000, "float32"))


@pytest.mark.parametrize("kind,g,dtype", CASES)
def test_col_stats_orders(kind, g, dtype):
    import torch

    lib = _lib.load()
    rng = np.random.default_rng(g)
    rows = _rows(kind, g, rng)
    idx = np.concatenate(rows).astype(np.int32)
    indptr = np.r_[0, np.cumsum([len(r) for r in rows])].astype(np.int64)
    vv = torch.from_numpy(rng.standard_normal(len(idx)).astype(np.float32)).to(getattr(torch, dtype)).cuda()
    val = vv.double().cpu().numpy()
    want = np.r_[np.bincount(idx, weights=val, minlength=g), np.bincount(idx, weights=val * val, minlength=g)]
    mag = np.r_[np.bincount(idx, weights=np.abs(val), minlength=g), want[g:]]
    code = {"float32": _lib.F32, "bfloat16": _lib.BF16, "float16": _lib.F16}[dtype]
    ip, ix = torch.from_numpy(indptr).cuda(), torch.from_numpy(idx).cuda()
    torch.cuda.synchronize()
    out = torch.full((2 * g,), float("nan"), dtype=torch.float64, device="cuda:0")
    x = _lib.Csr(len(rows), g, len(idx), ip.data_ptr(), ix.data_ptr(), vv.data_ptr(), code, _lib.MEM_DEVICE)
    err = _lib.errbuf()
    if g > _lib.NOALLOC_MAX_VARS:
        from scx_b200 import accel

        plan = accel.Plan(ip, ix, vv, (len(rows), g), n_components=2, n_oversamples=0)
        got = np.concatenate(plan.col_stats())
        plan.close()
    else:
        torch.cuda.synchronize()
        _lib.check(lib.scxpca_col_stats_noalloc(0, C.byref(x), C.c_void_p(out.data_ptr()), None, err, len(err)), err)
        got = out.cpu().numpy()
    assert np.all(np.abs(got - want) <= RTOL * np.maximum(mag, 1e-300))


@pytest.mark.parametrize("g", [3200, 3201, 4267, 6400, 6401, 12801, 30011])
def test_col_stats_of_wide_matrices(g):
    """Widths around those where fewer parts fit an SM and several warps share
    one, each with its own genes: a plan's sums, and the means of the same
    matrix uploaded from the host, whose statistics run in pieces and have the
    bits of one launch."""
    import torch

    from scx_b200 import accel

    rng = np.random.default_rng(g)
    rows = _rows("sorted", g, rng) + [np.arange(g), np.arange(0, g, 7), np.arange(g)[-40:]]
    idx = np.concatenate(rows).astype(np.int32)
    indptr = np.r_[0, np.cumsum([len(r) for r in rows])].astype(np.int64)
    val = rng.standard_normal(len(idx)).astype(np.float32)
    v64 = val.astype(np.float64)
    want = np.r_[np.bincount(idx, weights=v64, minlength=g), np.bincount(idx, weights=v64 * v64, minlength=g)]
    mag = np.r_[np.bincount(idx, weights=np.abs(v64), minlength=g), want[g:]]
    on_device = [torch.from_numpy(a).cuda() for a in (indptr, idx, val)]
    torch.cuda.synchronize()
    means = []
    for csr in (on_device, (indptr, idx, val)):
        plan = accel.Plan(*csr, (len(rows), g), n_components=2, n_oversamples=0, n_power_iterations=0)
        got = np.concatenate(plan.col_stats())
        assert np.all(np.abs(got - want) <= RTOL * np.maximum(mag, 1e-300))
        means.append(plan.run().mean)
        plan.close()
    assert np.array_equal(means[0], means[1])
