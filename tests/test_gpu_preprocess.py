"""Upstream producers on the device (needs a B200): normalize_total + log1p with
an optional per-row factor (scxpca_preprocess) and the mask_var column
projection (scxpca_project_columns), against the FP64 restatements in
oracle/rpca.py on the same raw counts.

Tolerances: values 1e-6 relative (the reference's own GPU-vs-CPU rtol for this
transform, scx-gpu/kernels/normalize_log1p.cu:10-15); the projection is integer
and byte work, so it is checked bit-exact; the PCA of the projected,
normalised matrix agrees with the oracle's PCA of the same pipeline to 1e-4 on
singular values (the strict-path parity bar).
"""

import numpy as np
import pytest

from oracle import rpca
from scx_b200 import accel

pytestmark = pytest.mark.gpu


def _raw_counts(n=3000, g=900, seed=0):
    rng = np.random.default_rng(seed)
    mu = rng.lognormal(-1.0, 1.5, g)
    size = rng.lognormal(0.0, 0.5, n)
    lam = np.outer(size, mu)
    counts = rng.negative_binomial(1 / 0.3, 1 / (1 + 0.3 * lam)).astype(np.float32)
    counts[7, :] = 0.0  # empty rows
    counts[11, :] = 0.0
    rr, cc = np.nonzero(counts)
    indptr = np.r_[0, np.cumsum(np.bincount(rr, minlength=n))].astype(np.int64)
    return rpca.Csr(indptr, cc.astype(np.int32), counts[rr, cc], (n, g))


def _dev(c):
    import torch
    return (torch.from_numpy(c.indptr).cuda(), torch.from_numpy(c.indices).cuda(),
            torch.from_numpy(np.ascontiguousarray(c.data, dtype=np.float32)).cuda())


@pytest.mark.parametrize("target_sum,log1p,factors", [(1e4, True, False), (1e4, False, False),
                                                      (None, True, False), (1e4, True, True)])
def test_normalize_log1p_matches_oracle(target_sum, log1p, factors):
    import torch

    c = _raw_counts()
    ip, ix, vv = _dev(c)
    rf = np.random.default_rng(1).uniform(0.5, 2.0, c.shape[0]).astype(np.float32) if factors else None
    got = accel.preprocess(ip, ix, vv, c.shape, target_sum=target_sum, log1p=log1p,
                           row_factors=None if rf is None else torch.from_numpy(rf).cuda())
    want = rpca.normalize_log1p(c, target_sum, log1p, rf)
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=1e-6, atol=0)
    # the input is untouched out of place; in place gives the same values
    np.testing.assert_array_equal(vv.cpu().numpy(), c.data)
    same = accel.preprocess(ip, ix, vv, c.shape, target_sum=target_sum, log1p=log1p,
                            row_factors=None if rf is None else torch.from_numpy(rf).cuda(), inplace=True)
    assert same.data_ptr() == vv.data_ptr()
    np.testing.assert_array_equal(vv.cpu().numpy(), got.cpu().numpy())


def test_project_columns_bit_exact():
    c = _raw_counts(seed=2)
    cols = np.flatnonzero(np.random.default_rng(3).random(c.shape[1]) < 0.3)
    ip, ix, vv = _dev(c)
    pip, pix, pvv, shape = accel.project_columns(ip, ix, vv, c.shape, cols)
    want = rpca.project_columns(c, cols)
    assert shape == want.shape
    np.testing.assert_array_equal(pip.cpu().numpy(), want.indptr)
    np.testing.assert_array_equal(pix.cpu().numpy(), want.indices)
    np.testing.assert_array_equal(pvv.cpu().numpy(), want.data)


def test_project_columns_rejects_bad_selections():
    c = _raw_counts(n=200, g=50, seed=4)
    ip, ix, vv = _dev(c)
    with pytest.raises(ValueError, match="sorted and unique"):
        accel.project_columns(ip, ix, vv, c.shape, [3, 2])
    with pytest.raises(ValueError, match="out of range"):
        accel.project_columns(ip, ix, vv, c.shape, [0, 50])


def test_raw_counts_to_pca_on_device_matches_oracle():
    """Raw counts resident on the device -> HVG column projection ->
    normalize_total(1e4) + log1p -> randomized PCA on the borrowed device CSR,
    against the oracle's run of the same pipeline with the same Omega."""
    c = _raw_counts(n=4000, g=1200, seed=5)
    cols = np.flatnonzero(np.random.default_rng(6).random(c.shape[1]) < 0.5)
    ip, ix, vv = _dev(c)
    pip, pix, pvv, shape = accel.project_columns(ip, ix, vv, c.shape, cols)
    accel.preprocess(pip, pix, pvv, shape, target_sum=1e4, log1p=True, inplace=True)
    k = 30
    om = rpca.gaussian_omega(shape[1], k, seed=0)
    res = accel.randomized_pca(pip, pix, pvv, shape, n_components=20, n_oversamples=10, n_power_iterations=4,
                               omega=om, math_mode="strict_fp32")
    pc = rpca.project_columns(c, cols)
    oc = pc.with_values(rpca.normalize_log1p(pc, 1e4, True))
    ref = rpca.randomized_pca(oc, 20, 10, 4, True, om)
    rel = np.abs(res.singular_values - ref["singular_values"]) / ref["singular_values"]
    assert rel.max() < 1e-4, rel.max()
    assert rpca.principal_angles(res.components.T, ref["components"].T).max() < 1e-3


@pytest.mark.parametrize("g", [800, 200_000])  # the column table in shared memory, and in global memory
def test_row_lengths_around_the_steps(g):
    """Rows around the 32-entry and 128-entry steps and around what a warp holds
    in registers (256 entries), projected bit for bit and normalised to the
    FP64 restatement (1e-6, the bound of this file)."""
    lengths = [0, 1, 31, 32, 33, 127, 128, 129, 255, 256, 257, 0, 700, 3]
    rng = np.random.default_rng(g)
    idx = np.concatenate([np.sort(rng.choice(g, m, replace=False)) for m in lengths]).astype(np.int32)
    idx[-1] = g - 1  # the last column of the last word
    c = rpca.Csr(np.r_[0, np.cumsum(lengths)].astype(np.int64), idx,
                 rng.integers(1, 50, len(idx)).astype(np.float32), (len(lengths), g))
    ip, ix, vv = _dev(c)
    got = accel.preprocess(ip, ix, vv, c.shape)
    np.testing.assert_allclose(got.cpu().numpy(), rpca.normalize_log1p(c, 1e4, True, None), rtol=1e-6, atol=0)
    for cols in ([g - 1], np.flatnonzero(rng.random(g) < 0.4), np.arange(g)):
        pip, pix, pvv, shape = accel.project_columns(ip, ix, vv, c.shape, cols)
        want = rpca.project_columns(c, np.asarray(cols))
        np.testing.assert_array_equal(pip.cpu().numpy(), want.indptr)
        np.testing.assert_array_equal(pix.cpu().numpy(), want.indices)
        np.testing.assert_array_equal(pvv.cpu().numpy(), want.data)


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 4096, 530_000])
def test_row_pointers_of_many_rows(n):
    """The projected row pointers are an exclusive scan in tiles of 2,048 rows
    (and 256 tiles a step): whole tiles, one row off them, more than one step."""
    per_row = np.random.default_rng(n).integers(0, 3, n)
    indptr = np.r_[0, np.cumsum(per_row)].astype(np.int64)
    starts = np.repeat(indptr[:-1], per_row)
    idx = (np.arange(indptr[-1]) - starts).astype(np.int32)
    c = rpca.Csr(indptr, idx, np.ones(len(idx), dtype=np.float32), (n, 40))
    ip, ix, vv = _dev(c)
    pip, pix, _, _ = accel.project_columns(ip, ix, vv, c.shape, [0, 39])
    np.testing.assert_array_equal(pip.cpu().numpy(), np.r_[0, np.cumsum(per_row > 0)])
    assert pix.numel() == (per_row > 0).sum() and not pix.any()


def test_producers_refuse_a_bad_csr():
    from scx_b200._lib import ScxPcaError

    c = _raw_counts(n=300, g=60, seed=8)
    for where, value, word in (("index", 60, "column index"), ("index", -1, "column index"), ("ptr", -5, "indptr"),
                               ("last", 1, "indptr")):
        ip, ix, vv = _dev(c)
        if where == "index":
            ix[ix.numel() - 1] = value
        else:
            at = 100 if where == "ptr" else len(ip) - 1
            ip[at] += value * 1000 if where == "ptr" else value
        for call in (lambda: accel.preprocess(ip, ix, vv, c.shape),
                     lambda: accel.project_columns(ip, ix, vv, c.shape, [1, 5])):
            with pytest.raises(ScxPcaError, match=word):
                call()


def test_counts_of_rows_of_a_million_entries():
    """Kept entries of rows that end around the most that is summed at once
    (2^20), and an index one past the columns as the last of the longest: refused."""
    from scx_b200._lib import ScxPcaError

    lengths = [(1 << 20) - 1, 1 << 20, (1 << 20) + 1, (1 << 20) + 300]
    g = max(lengths) + 40
    rng = np.random.default_rng(g)
    idx = np.concatenate([np.sort(rng.choice(g, m, replace=False)) for m in lengths]).astype(np.int32)
    c = rpca.Csr(np.r_[0, np.cumsum(lengths)].astype(np.int64), idx, np.arange(len(idx), dtype=np.float32),
                 (len(lengths), g))
    cols = np.flatnonzero(rng.random(g) < 0.3)
    keep = np.isin(idx, cols)
    ip, ix, vv = _dev(c)
    pip, pix, pvv, _ = accel.project_columns(ip, ix, vv, c.shape, cols)
    np.testing.assert_array_equal(pip.cpu().numpy(), np.r_[0, np.cumsum(keep)][c.indptr])
    np.testing.assert_array_equal(pix.cpu().numpy(), np.searchsorted(cols, idx[keep]))
    np.testing.assert_array_equal(pvv.cpu().numpy(), c.data[keep])
    ix[ix.numel() - 1] = g
    with pytest.raises(ScxPcaError, match="column index"):
        accel.project_columns(ip, ix, vv, c.shape, cols)


@pytest.mark.parametrize("n,where,value", [(300, "index", 60), (300, "index", -1), (5000, "ptr", -5000),
                                           (300, "last", 1), (0, "last", 2)])
def test_a_refused_projection_leaves_its_outputs(n, where, value):
    """The caller's row pointers and count are written for an accepted CSR only."""
    import ctypes as C

    import torch

    from scx_b200 import _lib

    c = _raw_counts(n=n or 300, g=60, seed=8)
    ip, ix, vv = _dev(c)
    if n == 0:
        ip, ix, vv = ip[:1].clone(), ix[:0], vv[:0]
    if where == "index":
        ix[ix.numel() - 1] = value
    else:
        ip[100 if where == "ptr" else len(ip) - 1] += value
    cols = np.array([1, 5], dtype=np.int32)
    out_ip = torch.full((n + 1,), -7, dtype=torch.int64, device="cuda")
    nnz = C.c_int64(-7)
    torch.cuda.synchronize()
    csr = _lib.Csr(n, 60, int(ix.numel()), ip.data_ptr(), ix.data_ptr(), vv.data_ptr(), _lib.F32, _lib.MEM_DEVICE)
    err = _lib.errbuf()
    st = _lib.load().scxpca_project_columns(0, C.byref(csr), cols.ctypes.data, 2, out_ip.data_ptr(), None, None,
                                            C.byref(nnz), None, err, len(err))
    assert st == _lib.INVALID_CSR
    assert nnz.value == -7
    assert (out_ip == -7).all()
