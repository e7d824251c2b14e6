"""The work this framework is used for, as timed cases.

Every case is one call (or one short chain of calls) of the public Python layer
on a seeded synthetic cells x genes matrix.  The matrix is what a PCA of
single-cell data meets: counts are Poisson around gene means that spread over
orders of magnitude (LogNormal(LOC, 1.5)), per-cell size factors
(LogNormal(0, 0.5)) and gene programs (modules of genes whose expression
follows a per-cell activity), stored as log1p(1e4 count / total).  About 9 % of
the entries are stored and their number differs by orders of magnitude from gene
to gene.  There are as many programs as components asked for, so the spectrum
has gaps down to the last component, and the components are defined well enough
for two runs to be compared.

The test matrix Omega is drawn here and handed to each call that takes one;
singular values are returned as float32, the precision of the products that
they come from, beside the embeddings and components.
"""

import math

import numpy as np
import torch

from scx_b200 import accel
from scx_b200.autograd import pca_scores

DEV = "cuda:0"
LOC = -2.8          # log-mean of the gene means: about 9 % of the entries stored
ACTIVITY = 1.5      # standard deviation of a program's log-activity
CELLS = 1_000_000   # most cells of a drawn case


def _pca_case(name, kind, n, g, nc, q, mode, qr="householder", center=True, scale=False, clip=0.0, values="f32"):
    return {"name": name, "kind": kind, "n_obs": n, "n_vars": g, "n_components": nc, "n_oversamples": 10,
            "n_power_iterations": q, "math_mode": mode, "qr_method": qr, "zero_center": center, "scale": scale,
            "clip_max": clip, "values": values}


def listed():
    return [
        # A small study (or a test set) on a resident plan, run again with another Omega:
        # nothing but launches and the latency of the small factorisations.
        _pca_case("run_fp32_2k", "run", 2_000, 500, 20, 2, "strict_fp32"),
        # The first call of most users: one sample of 10,000 cells, device arrays,
        # every option at its default, plan building included.
        _pca_case("pca_fp32_10k", "pca", 10_000, 2_000, 50, 2, "strict_fp32"),
        # The default precision at the size of a large study, matrix resident.
        _pca_case("run_fp32_250k", "run", 250_000, 2_000, 50, 2, "strict_fp32"),
        # The headline: an atlas of 1,000,000 cells on tensor cores, scaled and clipped.
        _pca_case("run_bf16_1m", "run", 1_000_000, 2_000, 50, 4, "mixed_bf16", "cholesky", True, True, 10.0),
        # An ordinary study on tensor cores, ragged sizes, few components, 16-bit input values.
        _pca_case("run_bf16_50k", "run", 50_021, 2_001, 30, 3, "mixed_bf16", values="bf16"),
        # A wide sketch (k = 110, two 64-column blocks) of more genes in FP16.
        _pca_case("run_f16_100pcs", "run", 120_000, 3_001, 100, 2, "mixed_f16"),
        # One call on a device matrix seen once: validation, statistics, scaling, packing and the PCA.
        _pca_case("pca_bf16_500k", "pca", 500_000, 2_000, 50, 4, "mixed_bf16", "cholesky", True, True, 10.0),
        # The same call on pinned host arrays, host embeddings back: the whole trip.
        _pca_case("host_bf16_100k", "host", 100_000, 2_000, 50, 2, "mixed_bf16", scale=True, clip=10.0),
        # A caller's own subspace iteration through the operator seam: product,
        # orthonormalisation, transposed product.
        _pca_case("step_fp32_50k", "step", 50_000, 2_000, 50, 0, "strict_fp32"),
        # One training step through the differentiable scores: forward and backward.
        _pca_case("grad_fp32_100k", "grad", 100_000, 2_000, 50, 4, "strict_fp32"),
        # Per-cluster PCAs of one atlas as one launch.
        {"name": "batch_bf16_64", "kind": "batch", "n_segments": 64, "n_vars": 2_000, "n_components": 30,
         "n_power_iterations": 3, "seed_sizes": 0},
        # The producers in front of a PCA: raw counts of all genes to normalised
        # log values of the selected ones, on the device.
        {"name": "counts_200k", "kind": "counts", "n_obs": 200_000, "n_vars": 6_000, "n_selected": 2_000},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["pca"] * 4 + ["host", "step", "step", "grad", "batch", "counts"])
    if kind == "batch":
        return {"kind": kind, "n_segments": rng.randint(8, 64), "n_vars": _log_uniform(rng, 500, 3_000),
                "n_components": rng.randint(10, 50), "n_power_iterations": rng.randint(2, 4),
                "seed_sizes": rng.randint(0, 999)}
    if kind == "counts":
        n = _log_uniform(rng, 5_000, 200_000)
        g = _log_uniform(rng, 2_000, 6_000)
        return {"kind": kind, "n_obs": n, "n_vars": g, "n_selected": rng.randint(500, g)}
    mode = rng.choice(["strict_fp32", "mixed_bf16", "mixed_bf16", "mixed_f16"])
    if kind in ("step", "grad"):
        mode = "strict_fp32"
    nc = rng.choice([rng.randint(10, 50), 50, rng.randint(51, 110)]) if kind != "grad" else rng.randint(10, 50)
    g = _log_uniform(rng, max(500, 12 * nc), 4_000)
    most = CELLS if mode != "strict_fp32" else 125_000
    if kind in ("host", "step", "grad"):
        most = 100_000
    n = _log_uniform(rng, 2_000, min(most, 2_000 * most // g))
    scale = kind != "grad" and rng.random() < 0.5
    c = _pca_case("", kind, n, g, nc, rng.randint(2, 4), mode, rng.choice(["householder", "cholesky"]), True, scale,
                  10.0 if scale else 0.0, "f32" if mode == "strict_fp32" or scale else rng.choice(["f32", mode[6:]]))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _counts(n, g, programs, seed):
    """(indptr int64, indices int32, counts float32) on the device.  Which cell
    expresses which gene is drawn from the sizes alone, so that every seed
    stores the same number of entries; the seed draws the order of the cells
    and the counts."""
    gen = torch.Generator(DEV).manual_seed(1_000_003 * n + g)
    weights = torch.pow(0.97, torch.arange(programs, device=DEV, dtype=torch.float32))
    module = torch.multinomial(weights, g, replacement=True, generator=gen)
    log_mu = LOC + 1.5 * torch.randn(g, device=DEV, generator=gen) - 0.5 * ACTIVITY ** 2
    per_row, cols, vals = [], [], []
    chunk = max(1, (1 << 27) // g)
    for r0 in range(0, n, chunk):
        m = min(chunk, n - r0)
        act = ACTIVITY * torch.randn((m, programs), device=DEV, generator=gen)
        size = 0.5 * torch.randn((m, 1), device=DEV, generator=gen)
        x = torch.poisson(act[:, module].add_(size).add_(log_mu).exp_(), generator=gen)
        at = x.nonzero()
        per_row.append(torch.bincount(at[:, 0], minlength=m))
        cols.append(at[:, 1].to(torch.int32))
        vals.append(x[at[:, 0], at[:, 1]])
        del x, at
    per_row, cols, vals = torch.cat(per_row), torch.cat(cols), torch.cat(vals)
    # the seed's order of the cells, and its counts
    gen = torch.Generator(DEV).manual_seed(seed)
    order = torch.randperm(n, device=DEV, generator=gen)
    begin = torch.cumsum(per_row, 0) - per_row
    per_row, begin = per_row[order], begin[order]
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(per_row, 0, out=indptr[1:])
    at = torch.arange(cols.numel(), device=DEV) + torch.repeat_interleave(begin - indptr[:-1], per_row)
    vals = vals[at]
    return indptr, cols[at], vals + torch.poisson(0.2 * vals, generator=gen)


def _log_values(indptr, counts):
    rows = torch.repeat_interleave(torch.diff(indptr))
    total = torch.zeros(indptr.numel() - 1, dtype=torch.float64, device=DEV)
    total.index_add_(0, rows, counts.double())
    return torch.log1p(1e4 * counts.double() / total[rows]).to(torch.float32)


_DTYPE = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}


def _width(c):
    return min(c["n_components"] + c.get("n_oversamples", 10), c["n_vars"], c["n_obs"])


def _matrix(c, seed):
    indptr, idx, counts = _counts(c["n_obs"], c["n_vars"], c["n_components"] + 2, seed)
    val = _log_values(indptr, counts).to(_DTYPE[c["values"]])
    torch.cuda.synchronize()  # a plan works on a stream of its own: its inputs have to be there
    return indptr, idx, val


def _gaussian(rows, cols, seed):
    gen = torch.Generator(DEV).manual_seed(7_919 * seed + 5)
    return torch.randn((cols, rows), device=DEV, generator=gen).t()  # (rows, cols), column-major


def _segments(c):
    rng = np.random.default_rng(c["seed_sizes"])
    sizes = np.clip(np.round(rng.lognormal(math.log(4_000), 1.0, c["n_segments"])), 500, 50_000).astype(np.int64)
    return np.concatenate([[0], np.cumsum(sizes)])


def _options(c):
    return dict(n_components=c["n_components"], n_oversamples=c["n_oversamples"],
                n_power_iterations=c["n_power_iterations"], zero_center=c["zero_center"], scale=c["scale"],
                clip_max=c["clip_max"] or None, qr_method=c["qr_method"], math_mode=c["math_mode"])


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        offsets = _segments(c)
        n = int(offsets[-1])
        indptr, idx, counts = _counts(n, c["n_vars"], c["n_components"] + 2, seed)
        val = _log_values(indptr, counts).to(torch.bfloat16)
        torch.cuda.synchronize()
        batch = accel.Batch(indptr, idx, val, (n, c["n_vars"]), offsets, n_components=c["n_components"],
                            n_power_iterations=c["n_power_iterations"], seed=seed, branches=-1)
        return {"kind": kind, "batch": batch, "out": torch.empty((n, c["n_components"]), device=DEV)}
    if kind == "counts":
        indptr, idx, counts = _counts(c["n_obs"], c["n_vars"], 50, seed)
        cols = np.sort(np.random.default_rng(c["n_vars"]).choice(c["n_vars"], c["n_selected"], replace=False))
        return {"kind": kind, "csr": (indptr, idx, counts), "shape": (c["n_obs"], c["n_vars"]),
                "cols": cols.astype(np.int32)}
    shape = (c["n_obs"], c["n_vars"])
    csr = _matrix(c, seed)
    omega = _gaussian(c["n_vars"], _width(c), seed)
    st = {"kind": kind, "csr": csr, "shape": shape, "omega": omega, "options": _options(c)}
    if kind in ("run", "step"):
        # a caller that mixes its own tensor operations with the seam's calls orders both on one stream
        st["stream"] = torch.cuda.Stream() if kind == "step" else None
        st["plan"] = accel.Plan(*csr, shape, stream=st["stream"].cuda_stream if kind == "step" else None,
                                **st["options"])
        st["out"] = torch.empty((c["n_obs"], c["n_components"]), device=DEV)
    elif kind == "host":
        st["pinned"] = [t.cpu().pin_memory() for t in csr]  # held: the arrays below are views of them
        st["csr"] = [t if t.dtype == torch.bfloat16 else t.numpy() for t in st["pinned"]]
        st["omega"] = omega.cpu().numpy()
        st["pinned_out"] = torch.empty((c["n_obs"], c["n_components"]), pin_memory=True)
        st["out"] = st["pinned_out"].numpy()
    elif kind == "grad":
        indptr, idx, val = csr
        mean = torch.zeros(c["n_vars"], device=DEV, dtype=torch.float64)
        mean.index_add_(0, idx.long(), val.double())
        mean /= c["n_obs"]
        gen = torch.Generator(DEV).manual_seed(31 * seed + 3)
        st["values"] = val.requires_grad_(True)
        st["center"] = mean.float().requires_grad_(True)
        st["gene_scale"] = torch.ones(c["n_vars"], device=DEV).requires_grad_(True)
        st["weight"] = torch.randn((c["n_obs"], c["n_components"]), device=DEV, generator=gen)
        torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _of_result(r):
    return {"embeddings": r.embeddings, "components": r.components,
            "singular_values": r.singular_values.astype(np.float32)}


def run(state):
    s, kind = state, state["kind"]
    if kind == "run":
        return _of_result(s["plan"].run(omega=s["omega"], embeddings_out=s["out"]))
    if kind == "pca":
        return _of_result(accel.randomized_pca(*s["csr"], s["shape"], omega=s["omega"], device_embeddings=True,
                                               **s["options"]))
    if kind == "host":
        return _of_result(accel.randomized_pca(*s["csr"], s["shape"], omega=s["omega"], embeddings_out=s["out"],
                                               **s["options"]))
    if kind == "step":
        with torch.cuda.stream(s["stream"]):
            y = s["plan"].matmat(s["omega"])
            q = s["plan"].qr(y.clone())
            return {"y": y, "q": q, "v": s["plan"].rmatmat(q).float()}
    if kind == "grad":
        o = s["options"]
        scores = pca_scores(s["csr"][0], s["csr"][1], s["values"], s["shape"], center=s["center"],
                            scale=s["gene_scale"], omega=s["omega"], n_components=o["n_components"],
                            n_oversamples=o["n_oversamples"], n_power_iterations=o["n_power_iterations"],
                            qr_method=o["qr_method"])
        loss = (s["weight"] * scores * scores).sum()
        gv, gc, gs = torch.autograd.grad(loss, [s["values"], s["center"], s["gene_scale"]])
        return {"scores": scores.detach(), "grad_values": gv, "grad_center": gc, "grad_scale": gs}
    if kind == "batch":
        emb, comps, sv, _, _ = s["batch"].run(embeddings_out=s["out"])
        return {"embeddings": emb, "components": comps, "singular_values": sv.astype(np.float32)}
    indptr, idx, val, shape = accel.project_columns(*s["csr"], s["shape"], s["cols"])
    return {"indptr": indptr, "indices": idx, "values": accel.preprocess(indptr, idx, val, shape, inplace=True)}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _stored(n, g):
    return 0.09 * n * g


def work(case):
    c, kind = case, case["kind"]
    g = c["n_vars"]
    if kind == "counts":
        nnz = _stored(c["n_obs"], g)
        kept = nnz * c["n_selected"] / g
        return {"bytes": 8.0 * nnz + 8.0 * kept + 16.0 * c["n_obs"], "flops": 4.0 * kept}
    n = int(_segments(c)[-1]) if kind == "batch" else c["n_obs"]
    segments = c["n_segments"] if kind == "batch" else 1
    nnz, nc = _stored(n, g), c["n_components"]
    k = nc + 10
    value_bytes = 2 if kind == "batch" or c["values"] != "f32" else 4
    matrix = nnz * (4 + value_bytes) + 8.0 * n
    product, gram = 2.0 * nnz * k, 1.0 * n * k * k
    if kind == "step":
        return {"bytes": matrix + 4.0 * n * k * 2 + 4.0 * g * k * 2, "flops": 2 * product + 2 * gram + n * k * k}
    q = c["n_power_iterations"]
    flops = 2 * (q + 1) * product + (q + 2) * gram + 2.0 * n * k * k + 2.0 * n * k * nc
    total = matrix + 4.0 * n * nc + 4.0 * segments * g * nc
    if kind == "grad":  # H, X~ A and 8 solve steps of two products; the sampled rank-2c gradient
        flops += 2 * product + 16 * product + 4.0 * nnz * nc
        total += 4.0 * nnz + 4.0 * n * nc
    return {"bytes": total, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _dense(csr, shape):
    indptr, idx, val = (torch.as_tensor(t).to(DEV).detach() for t in csr)
    x = torch.zeros(shape, dtype=torch.float64, device=DEV)
    x[torch.repeat_interleave(torch.diff(indptr)), idx.long()] = val.double()
    return x


def _standardised(c, csr):
    x = _dense(csr, (c["n_obs"], c["n_vars"]))
    x -= x.mean(0)
    if c["scale"]:
        sd = x.square().sum(0).div_(max(c["n_obs"] - 1, 1)).sqrt_()
        x /= torch.where(sd == 0, torch.ones_like(sd), sd)
        if c["clip_max"]:
            x.clamp_(-c["clip_max"], c["clip_max"])
        x -= x.mean(0)
    return x


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("batch", "grad"):
        return None  # the batch draws its own Omega; the gradient of a randomized PCA has no closed form to hold it to
    if kind == "counts":
        s = prepare(c, seed)
        kept = _dense(s["csr"], s["shape"])[:, torch.as_tensor(s["cols"], device=DEV).long()]
        at = kept.nonzero()
        total = kept.sum(1, keepdim=True)
        logs = torch.log1p(kept * (1e4 / torch.where(total > 0, total, torch.ones_like(total))))
        indptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), torch.cumsum((kept != 0).sum(1), 0)])
        return {"indptr": indptr, "indices": at[:, 1].to(torch.int32), "values": logs[at[:, 0], at[:, 1]]}
    csr = _matrix(c, seed)
    x = _standardised(c, csr)
    y = x @ _gaussian(c["n_vars"], _width(c), seed).double()
    if kind == "step":
        r = torch.linalg.cholesky(y.t() @ y).t()
        q = torch.linalg.solve_triangular(r, y, upper=True, left=False)
        return {"y": y, "q": q, "v": x.t() @ q}
    q = torch.linalg.qr(y).Q
    for _ in range(c["n_power_iterations"]):
        z = torch.linalg.qr(x.t() @ q).Q
        q = torch.linalg.qr(x @ z).Q
    sv = torch.linalg.svdvals(x.t() @ q)
    # components and embeddings are defined up to the sign of each component
    return {"embeddings": None, "components": None, "singular_values": sv[: c["n_components"]]}
