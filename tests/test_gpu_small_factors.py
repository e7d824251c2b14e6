"""The k x k factorisations at the edges of their panels (needs a B200).

The Cholesky takes rows in panels of eight on a 64- or 128-wide tile, the
eigensolver columns in pairs on the same two widths: every remainder of the
panel, the widest and narrowest of each tile, and the odd k with its dummy
column.  The Q factor against the FP64 Cholesky factor of the same Gram
(Q = A R^{-1}, R with a positive diagonal): A is random with cond(A) < 10, so
FP32 storage of Q and of the two intermediate passes leaves about 3 * 6e-8 of
an entry's size.  Singular values against the FP64 oracle as in the parity tests.
"""

import numpy as np
import pytest

from oracle import rpca
from scx_b200 import accel
from scx_b200.synth import synth_nb_csr

pytestmark = pytest.mark.gpu

WIDTHS = (1, 2, 7, 8, 9, 24, 31, 57, 63, 64, 65, 72, 97, 120, 127, 128)


@pytest.fixture(scope="module")
def matrix():
    n, g = 700, 200
    indptr, idx, val = synth_nb_csr(n, g, seed=11, loc=-1.5)
    return rpca.Csr(indptr, idx, val, (n, g))


@pytest.mark.parametrize("k", WIDTHS)
@pytest.mark.parametrize("method", ("cholesky", "householder"))
def test_qr_factor_widths(matrix, k, method):
    import torch

    c = matrix
    plan = accel.Plan(c.indptr, c.indices, c.data, c.shape, n_components=k, n_oversamples=0, qr_method=method)
    a = np.random.default_rng(k).standard_normal((700, k)).astype(np.float32)
    q = plan.qr(torch.from_numpy(a).cuda()).cpu().numpy().astype(np.float64)
    plan.close()
    a64 = a.astype(np.float64)
    r = np.linalg.cholesky(a64.T @ a64).T
    want = np.linalg.solve(r.T, a64.T).T
    assert np.abs(q - want).max() < 2e-6 * np.abs(want).max()
    assert np.abs(q.T @ q - np.eye(k)).max() < 2e-6


@pytest.mark.parametrize("k", WIDTHS)
def test_singular_values_widths(matrix, k):
    c = matrix
    om = np.random.default_rng(100 + k).standard_normal((200, k))
    ref = rpca.randomized_pca(c, k, 0, 1, True, om)
    res = accel.randomized_pca(c.indptr, c.indices, c.data, c.shape, n_components=k, n_oversamples=0,
                               n_power_iterations=1, omega=om)
    rel = np.abs(res.singular_values - ref["singular_values"]) / ref["singular_values"]
    assert rel.max() < 1e-4
    assert np.abs(res.components @ res.components.T - np.eye(k)).max() < 1e-5


@pytest.mark.parametrize("m", (128, 129, 130, 131, 1187, 9473))  # 9,473 rows: 32 a block, and one over
@pytest.mark.parametrize("k", (20, 60, 90, 128))
def test_qr_row_counts(matrix, m, k):
    """The Gram behind a factor takes four rows at a time, a row group per block:
    every remainder, blocks with no row, one row over.  The bound of
    test_qr_factor_widths; the square case (m = k = 128) only keeps its
    columns orthogonal, cond(A)^2 being past FP32 there."""
    import torch

    c = matrix
    plan = accel.Plan(c.indptr, c.indices, c.data, c.shape, n_components=k, n_oversamples=0)
    a = np.random.default_rng(m + k).standard_normal((m, k)).astype(np.float32)
    q = plan.qr(torch.from_numpy(a).cuda()).cpu().numpy().astype(np.float64)
    plan.close()
    assert np.abs(q.T @ q - np.eye(k)).max() < 2e-6
    if m > 2 * k:
        a64 = a.astype(np.float64)
        r = np.linalg.cholesky(a64.T @ a64).T
        want = np.linalg.solve(r.T, a64.T).T
        assert np.abs(q - want).max() < 2e-6 * np.abs(want).max() * np.linalg.cond(a64)


@pytest.mark.parametrize("n,g,nc,over", [
    (300, 20, 5, 15),      # ld 32; components end inside the first half of the columns
    (300, 64, 33, 31),     # both halves
    (400, 95, 95, 0),      # ld 96, as many components as columns
    (500, 127, 70, 57),    # ld 128
    (32, 5003, 9, 22),     # more strips of genes than blocks, a ragged last one
    (120, 4801, 65, 54),
])
def test_finish_is_consistent(n, g, nc, over):
    """A sketch as wide as the centred matrix's rank spans its range, so the
    embeddings are the matrix times the components, and these are orthonormal:
    FP32 factors of a well-conditioned sketch, 2e-5 of the largest singular value."""
    rng = np.random.default_rng(n + g)
    x = rng.standard_normal((n, g)).astype(np.float32) * (rng.random((n, g)) < 0.4)
    rows, cols = np.nonzero(x)
    indptr = np.r_[0, np.cumsum(np.bincount(rows, minlength=n))]
    res = accel.randomized_pca(indptr, cols.astype(np.int32), x[rows, cols], (n, g), n_components=nc,
                               n_oversamples=over, n_power_iterations=2)
    xc = x.astype(np.float64) - x.astype(np.float64).mean(axis=0)
    comps = np.asarray(res.components, dtype=np.float64)
    emb = np.asarray(res.embeddings, dtype=np.float64)
    s = np.linalg.svd(xc, compute_uv=False)[:nc]
    assert np.abs(comps @ comps.T - np.eye(nc)).max() < 2e-5
    assert np.abs(res.singular_values - s).max() < 2e-5 * s[0]
    assert np.abs(emb - xc @ comps.T).max() < 2e-5 * s[0]
