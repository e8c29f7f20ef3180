"""Performance cases of the package: what a user has it compute, at the sizes it is used at.

The listed cases stand for the work of a GWAS on this package, through its public calls:

* association of one chunk of SNPs against a resident cohort (``engine.DeviceCohort`` with
  ``engine.ChunkGraph`` or, eagerly, ``decode_packed`` and ``associate_codes``), in both
  precisions, every test mode, one or many phenotypes, one to four covariate columns, with
  and without missing calls and dropped samples;
* the set-up of a cohort for new phenotypes on a resident eigendecomposition;
* kinship matrices, from memory and from a .bed file, in both precisions;
* the whole streaming call, from a .bed file and a kinship matrix to the result records
  (this one contains the eigendecomposition).

Genotypes are drawn as ``jamma_b200.synth`` draws them: Binomial(2, p), p ~ U(0.05, 0.5),
independent missing calls.  Cohorts of association cases have a closed-form orthonormal
eigenbasis (a Hartley matrix with permuted, sign-flipped rows) and a skewed spectrum with
one zero eigenvalue, so that no eigendecomposition is needed to prepare them.
"""

from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from jamma_b200 import compute_centered_kinship, compute_kinship_from_bed, run_lmm_association_streaming
from jamma_b200 import engine as eng
from jamma_b200 import synth
from jamma_b200.io import write_plink_records
from jamma_b200.kinship import snp_stats_from_counts


def _assoc(name, n, m, c, phi, mode, precision, missing, graph=True, dropped=0):
    case = {"kind": "assoc", "n": n, "m": m, "c": c, "phi": phi, "mode": mode,
            "precision": precision, "missing": missing, "graph": graph, "dropped": dropped}
    return case if name is None else {"name": name, **case}


def listed() -> list[dict]:
    return [
        # the smallest call: the cohort of the smoke test, default precision, issued eagerly
        _assoc("assoc_smoke_fp64", 500, 500, 1, 1, 1, "fp64", 0.01, graph=False),
        # a mouse cohort (n = 1940), Wald tests, default precision: the commonest analysis
        _assoc("assoc_mouse_fp64", 1940, 8192, 1, 1, 1, "fp64", 0.01),
        # n = 10 000 with covariates, every test, default precision
        _assoc("assoc_covariates_fp64", 10000, 2048, 3, 1, 4, "fp64", 0.01),
        # the headline size in the default precision
        _assoc("assoc_full_fp64", 20000, 2048, 1, 1, 4, "fp64", 0.01),
        # the headline workload: n = 20 000, every test, mixed precision, chunks of 8192 SNPs
        _assoc("assoc_headline_mixed", 20000, 8192, 1, 1, 4, "mixed", 0.01),
        # the batched configuration: 64 phenotypes at once
        _assoc("assoc_batched_mixed", 20000, 2048, 1, 64, 4, "mixed", 0.01),
        # a job of the serving mix: odd cohort size, some samples without phenotypes, a few
        # phenotypes, covariates, likelihood-ratio tests
        _assoc("assoc_serving_mixed", 5003, 8000, 2, 4, 2, "mixed", 0.01, dropped=98),
        # new phenotypes on a resident cohort: the set-up that a served job waits for
        {"name": "cohort_setup_mixed", "kind": "cohort", "n": 20000, "c": 1, "phi": 4, "mode": 4,
         "precision": "mixed"},
        # kinship of a genotype matrix in memory, default precision
        {"name": "kinship_memory_fp64", "kind": "kin_mem", "n": 1000, "m": 10000,
         "precision": "fp64", "missing": 0.01},
        # kinship streamed from a .bed file, default precision, odd sample count
        {"name": "kinship_bed_fp64", "kind": "kin_bed", "n": 8001, "m": 20000,
         "precision": "fp64", "missing": 0.01},
        # the INT8 form at the headline cohort size (a part of its SNPs, ragged)
        {"name": "kinship_bed_int8", "kind": "kin_bed", "n": 20000, "m": 30011,
         "precision": "int8", "missing": 0.01},
        # the whole call on the mouse cohort: .bed file and kinship matrix in, records out
        {"name": "runner_mouse_fp64", "kind": "runner", "n": 1940, "m": 12226, "c": 1, "mode": 1,
         "precision": "fp64", "missing": 0.01},
    ]


def _log_int(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["fp64", "fp64", "mixed", "mixed", "mixed", "cohort", "kin_mem", "kin_bed",
                       "kin_bed", "runner"])
    missing = rng.choice([0.0, 0.002, 0.01, 0.01, 0.02])
    if kind == "fp64":
        n = _log_int(rng, 200, 12000)
        m = min(_log_int(rng, 64, 8192), max(64, int(2e11 / n**2)))
        phi = rng.choice([1, 1, 1, 2, 3])
        return _assoc(None, n, m, rng.choice([1, 1, 2, 3, 4]), phi, rng.randint(1, 4), "fp64", missing,
                      graph=rng.random() < 0.8, dropped=rng.choice([0, 0, n // 50]))
    if kind == "mixed":
        n = _log_int(rng, 700, 20000)
        phi = rng.choice([1, 1, 2, 4, 8, 30, 64])
        if 97 * (4 + phi) > n:
            phi = 1
        m = min(_log_int(rng, 256, 8192), 131072 // phi)
        return _assoc(None, n, m, rng.choice([1, 1, 2, 3, 4]), phi, rng.randint(1, 4), "mixed", missing,
                      graph=rng.random() < 0.8, dropped=rng.choice([0, 0, n // 50]))
    if kind == "cohort":
        return {"kind": "cohort", "n": _log_int(rng, 1000, 16000), "c": rng.choice([1, 2, 3]),
                "phi": rng.choice([1, 2, 4, 8]), "mode": rng.randint(1, 4),
                "precision": rng.choice(["fp64", "mixed"])}
    if kind == "kin_mem":
        return {"kind": "kin_mem", "n": _log_int(rng, 100, 2000), "m": _log_int(rng, 500, 8000),
                "precision": rng.choice(["fp64", "fp64", "int8"]), "missing": missing}
    if kind == "kin_bed":
        n = _log_int(rng, 500, 16000)
        return {"kind": "kin_bed", "n": n, "m": _log_int(rng, 2000, min(40000, int(3.2e8 / n))),
                "precision": rng.choice(["fp64", "int8"]), "missing": missing}
    return {"kind": "runner", "n": _log_int(rng, 300, 2500), "m": _log_int(rng, 1000, 16000),
            "c": rng.choice([1, 2, 3]), "mode": rng.randint(1, 4),
            "precision": rng.choice(["fp64", "mixed"]), "missing": missing}


# ---------------------------------------------------------------- inputs
def _basis(n: int, rng) -> torch.Tensor:
    """Orthonormal eigenvectors, one per row (the column-major layout of the package)."""
    perm = torch.from_numpy(rng.permutation(n)).to("cuda")
    sign = torch.from_numpy(rng.choice([-1.0, 1.0], n)).to("cuda")
    U = torch.empty((n, n), dtype=torch.float64, device="cuda")
    step = max(1, 40_000_000 // n)
    for s in range(0, n, step):
        k = torch.arange(s, min(n, s + step), device="cuda")
        ang = ((k[:, None] * perm[None, :]) % n).to(torch.float64) * (2.0 * math.pi / n)
        U[s:s + k.numel()] = (torch.cos(ang) + torch.sin(ang)) * sign / math.sqrt(n)
    return U


def _cohort_inputs(case, seed):
    """(U, eigenvalues, covariates, phenotypes): eigenvectors and values on the device, the
    others on the host."""
    n, c, phi = case["n"], case["c"], case["phi"]
    rng = np.random.default_rng([seed, n, c, phi])
    U = _basis(n, rng)
    ev = np.sort(0.3 * np.exp(0.8 * rng.standard_normal(n)))
    ev[0] = 0.0
    evals = torch.from_numpy(ev).to("cuda")
    W = np.column_stack([np.ones(n), rng.standard_normal((n, c - 1))])
    h2 = rng.uniform(0.1, 0.7, phi)
    g = torch.from_numpy(rng.standard_normal((phi, n)) * np.sqrt(ev / ev.mean())).to("cuda")
    g = (g @ U).cpu().numpy().T * np.sqrt(h2 / (1.0 - h2))
    y = g + rng.standard_normal((n, phi)) + 0.3 * W[:, -1:]
    return U, evals, W, y


def _records(case, seed):
    """Packed records on the device, the analysed samples (None: all) and the float32
    means that the streaming path imputes with."""
    n, m = case["n"], case["m"]
    n_file = n + case.get("dropped", 0)
    packed = synth.packed_records_device(n_file, m, case["missing"], seed)
    sidx = None
    if n_file != n:
        keep = np.sort(np.random.default_rng([seed, 7]).permutation(n_file)[:n])
        sidx = torch.from_numpy(keep.astype(np.int32)).to("cuda")
    _, counts = eng.decode_packed(packed, n_file, sidx, n)
    mean, miss, _ = snp_stats_from_counts(counts.cpu().numpy(), n, np.float32)
    return packed, sidx, mean.astype(np.float64), bool(np.any(miss > 0))


class _Files:
    """A PLINK fileset in a temporary folder that goes when the state goes."""

    def __init__(self, packed: torch.Tensor, n: int):
        self.dir = tempfile.TemporaryDirectory(prefix="jamma_perf_")
        self.prefix = os.path.join(self.dir.name, "cohort")
        write_plink_records(self.prefix, packed.cpu().numpy(), n)


def _imputed(packed, n, sidx=None) -> torch.Tensor:
    """(m, n) float64 genotypes, missing calls replaced by the float64 mean."""
    b = packed
    two = torch.stack([b & 3, (b >> 2) & 3, (b >> 4) & 3, b >> 6], 2).reshape(b.shape[0], -1)
    two = two[:, :n] if sidx is None else two[:, sidx.long()]
    g = torch.tensor([2.0, math.nan, 1.0, 0.0], dtype=torch.float64, device=b.device)[two.long()]
    mean = torch.nanmean(g, 1, keepdim=True)
    return torch.where(torch.isnan(g), mean, g)


def _kinship(packed, n) -> torch.Tensor:
    K = torch.zeros((n, n), dtype=torch.float64, device=packed.device)
    step = max(1, 60_000_000 // n)
    for s in range(0, packed.shape[0], step):
        x = _imputed(packed[s:s + step], n)
        x -= x.mean(1, keepdim=True)
        K.addmm_(x.T, x)
    return K / packed.shape[0]


def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind == "assoc":
        U, evals, W, y = _cohort_inputs(case, seed)
        packed, sidx, means, has_missing = _records(case, seed)
        cohort = eng.DeviceCohort(evals, U, W, y, case["mode"], precision=case["precision"])
        means = torch.from_numpy(means).to("cuda")
        n_file = case["n"] + case["dropped"]
        graph = None
        if case["graph"]:
            graph = eng.ChunkGraph(cohort, case["m"], n_file, sidx, has_missing=has_missing)
        return {"case": case, "cohort": cohort, "packed": packed, "sidx": sidx, "means": means,
                "n_file": n_file, "missing": has_missing, "graph": graph}
    if kind == "cohort":
        U, evals, W, y = _cohort_inputs(case, seed)
        planes = eng.ozaki_split(U) if case["precision"] == "mixed" else None
        return {"case": case, "U": U, "evals": evals, "W": W, "y": y, "planes": planes}
    packed = synth.packed_records_device(case["n"], case["m"], case["missing"], seed)
    if kind == "kin_mem":
        b = packed
        two = torch.stack([b & 3, (b >> 2) & 3, (b >> 4) & 3, b >> 6], 2).reshape(b.shape[0], -1)
        g = torch.tensor([2.0, math.nan, 1.0, 0.0], dtype=torch.float64, device=b.device)[two.long()]
        return {"case": case, "g": g[:, :case["n"]].T.contiguous().cpu().numpy()}
    if kind == "kin_bed":
        return {"case": case, "files": _Files(packed, case["n"])}
    n = case["n"]
    K = _kinship(packed, n)
    rng = np.random.default_rng([seed, n, 3])
    W = np.column_stack([np.ones(n), rng.standard_normal((n, case["c"] - 1))])
    g = torch.linalg.cholesky(K + 0.02 * torch.eye(n, dtype=torch.float64, device="cuda"))
    g = (g @ torch.from_numpy(rng.standard_normal(n)).to("cuda")).cpu().numpy()
    y = g / g.std() * rng.uniform(0.4, 1.2) + rng.standard_normal(n) + 0.3 * W[:, -1]
    return {"case": case, "files": _Files(packed, n), "K": K.cpu().numpy(), "W": W, "y": y}


# ---------------------------------------------------------------- one pass
_RECORD = {1: ("beta", "se", "logl_H1", "l_remle", "p_wald"), 2: ("l_mle", "p_lrt"),
           3: ("beta", "se", "p_score"),
           4: ("beta", "se", "logl_H1", "l_remle", "p_wald", "p_score", "l_mle", "p_lrt")}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "assoc":
        if state["graph"] is not None:  # one chunk as the streaming runner replays it
            graph = state["graph"]
            graph.packed.copy_(state["packed"], non_blocking=True)
            graph.means.copy_(state["means"], non_blocking=True)
            return graph.replay()
        cohort = state["cohort"]
        codes, _ = eng.decode_packed(state["packed"], state["n_file"], state["sidx"], case["n"],
                                     cohort.code_ld)
        return cohort.associate_codes(codes, state["means"], has_missing=state["missing"])
    if kind == "cohort":
        c = eng.DeviceCohort(state["evals"], state["U"], state["W"], state["y"], case["mode"],
                             precision=case["precision"], ozaki=state["planes"])
        out = {"UtW": c.UtW, "Uty": c.Uty}
        if c.lam0 is not None:
            out.update(lam0=c.lam0, logl0=c.logl0)
        return out
    if kind == "kin_mem":
        return compute_centered_kinship(state["g"], precision=case["precision"])
    if kind == "kin_bed":
        return compute_kinship_from_bed(state["files"].prefix, as_device=True,
                                        precision=case["precision"])
    rows = run_lmm_association_streaming(state["files"].prefix, state["y"], kinship=state["K"],
                                         covariates=state["W"], lmm_mode=case["mode"],
                                         precision=case["precision"])
    return {k: np.array([getattr(r, k) for r in rows], dtype=np.float64)
            for k in ("af", *_RECORD[case["mode"]])}


def work(case: dict) -> dict:
    n, kind = case["n"], case["kind"]
    if kind == "assoc":
        # rotation U^T G, then one weighted reduction of every column pair with each SNP for
        # the grid of 50 lambdas; U and the records are read, the statistics written once
        c, phi, m = case["c"], case["phi"], case["m"]
        return {"bytes": 8.0 * n * n + m * (n / 4 + 8) + 8.0 * n * (c + phi) + 40.0 * m * phi,
                "flops": 2.0 * n * n * m + 100.0 * n * m * (c + phi + 1)}
    if kind == "cohort":
        k = case["c"] + case["phi"]
        return {"bytes": 8.0 * n * n + 32.0 * n * k,
                "flops": 2.0 * n * n * k * (98 if case["precision"] == "mixed" else 1)}
    m = case["m"]
    kin = {"bytes": m * n / 4 + 8.0 * n * n, "flops": 1.0 * n * n * m}
    if kind == "kin_mem":
        return {"bytes": 8.0 * m * n + 8.0 * n * n, "flops": kin["flops"]}
    if kind == "kin_bed":
        return kin
    return {"bytes": 16.0 * n * n + m * n / 4 + 60.0 * m, "flops": 9.0 * n**3 + 2.0 * n * n * m}


# ---------------------------------------------------------------- 64-bit values
_PHI = 0.6180339887498949


def _pab(rows, c):
    """Project the c covariates, then the genotype, out of the weighted Gram entries
    rows[(a, b)] (a <= b; a, b < c covariates, c genotype, c + 1 phenotype).  Returns the
    pivots, (xx, xy, yy) after the covariates and yy after the genotype as well."""
    r = dict(rows)
    pivots = []
    for p in range(c + 1):
        if p == c:
            level = (r[c, c], r[c, c + 1], r[c + 1, c + 1])
        pivots.append(r[p, p])
        inv = torch.where(r[p, p] != 0, 1.0 / r[p, p], torch.zeros_like(r[p, p]))
        r = {(a, b): v - r[p, a] * r[p, b] * inv for (a, b), v in r.items() if a > p}
    return pivots, level, r[c + 1, c + 1]


class _Exact:
    """The search and the statistics of one phenotype over a block of rotated genotypes."""

    def __init__(self, ev, W, y, X, l_min=1e-5, l_max=1e5, n_grid=50, n_iter=20):
        self.ev, self.W, self.y, self.X = ev, W, y, X
        self.n, self.c = ev.numel(), W.shape[0]
        self.df = self.n - self.c - 1
        self.grid = torch.linspace(math.log(l_min), math.log(l_max), n_grid, dtype=torch.float64,
                                   device=ev.device)
        self.n_iter = n_iter

    def sums(self, lam):
        """Weighted Gram entries and log|H| at one lambda per SNP (or one for all)."""
        v = lam[:, None] * self.ev + 1.0
        h = 1.0 / v
        cols, c = [*self.W, None, self.y], self.c
        hx = h * self.X
        rows = {}
        for a in range(c + 2):
            for b in range(a, c + 2):
                if a == c and b == c:
                    rows[a, b] = (hx * self.X).sum(1)
                elif a == c or b == c:
                    rows[a, b] = hx @ (cols[b] if a == c else cols[a])
                else:
                    rows[a, b] = (h @ (cols[a] * cols[b])).expand(self.X.shape[0])
        return rows, torch.log(v.abs()).sum(1).expand(self.X.shape[0])

    def logl(self, s, reml):
        rows, logdet = self.sums(torch.exp(s))
        pivots, level, yy1 = _pab(rows, self.c)
        pyy = torch.where((yy1 >= 0) & (yy1 < 1e-8), torch.full_like(yy1, 1e-8), yy1)
        k = self.df if reml else self.n
        f = 0.5 * k * (math.log(k) - math.log(2 * math.pi) - 1.0) - 0.5 * logdet
        if reml:
            ones, _ = self.sums(torch.zeros(1, dtype=torch.float64, device=s.device))
            iab, _, _ = _pab(ones, self.c)
            f = f - 0.5 * sum(torch.log(p) - torch.log(q) for p, q in zip(pivots, iab))
        return f - 0.5 * k * torch.log(pyy), level, pyy

    def search(self, reml):
        vals = torch.stack([self.logl(g.reshape(1), reml)[0] for g in self.grid])
        best = vals.argmax(0)
        last = self.grid.numel() - 1
        a, b = self.grid[(best - 1).clamp(min=0)], self.grid[(best + 1).clamp(max=last)]
        c, d = b - _PHI * (b - a), a + _PHI * (b - a)
        fc, fd = self.logl(c, reml)[0], self.logl(d, reml)[0]
        for _ in range(self.n_iter):
            left = fc > fd
            a, b = torch.where(left, a, c), torch.where(left, d, b)
            c, d = b - _PHI * (b - a), a + _PHI * (b - a)
            f = self.logl(torch.where(left, c, d), reml)[0]
            fc, fd = torch.where(left, f, fd), torch.where(left, fc, f)
        s = 0.5 * (a + b)
        return s, *self.logl(s, reml)


def _null_model(ev, W, y):
    """(lambda, log-likelihood) of the model without a genotype (always the default range)."""
    n, c = ev.numel(), W.shape[0]
    cols = [*W, y]

    def neg(s):
        v = math.exp(s) * ev + 1.0
        h = 1.0 / v
        rows = {(a, b): (h * cols[a] * cols[b]).sum() for a in range(c + 1) for b in range(a, c + 1)}
        for p in range(c):
            rows = {(a, b): x - rows[p, a] * rows[p, b] / rows[p, p]
                    for (a, b), x in rows.items() if a > p}
        pyy = max(float(rows[c, c]), 1e-8)
        return -(0.5 * n * (math.log(n) - math.log(2 * math.pi) - 1.0)
                 - 0.5 * float(torch.log(v.abs()).sum()) - 0.5 * n * math.log(pyy))

    lo, hi, num = math.log(1e-5), math.log(1e5), 50
    step = (hi - lo) / (num - 1)
    best = int(np.argmin([neg(lo + i * step) for i in range(num)]))
    a, b = lo + max(best - 1, 0) * step, lo + min(best + 1, num - 1) * step
    c1, d1 = b - _PHI * (b - a), a + _PHI * (b - a)
    fc, fd = neg(c1), neg(d1)
    for _ in range(20):
        if fc < fd:
            b, d1, fd = d1, c1, fc
            c1 = b - _PHI * (b - a)
            fc = neg(c1)
        else:
            a, c1, fc = c1, d1, fd
            d1 = a + _PHI * (b - a)
            fd = neg(d1)
    s = 0.5 * (a + b)
    return math.exp(s), -neg(s)


def _f_sf(f, df):
    """P(F(1, df) > f) = I_z(df/2, 1/2), z = df/(df + f), by the continued fraction of
    DLMF 8.17.22 in the form for z near 1: 1 - I_{1-z}(1/2, df/2), or directly."""
    a = 0.5 * df
    big, ratio = a, 1.0  # Gamma(a + 1/2) / Gamma(a): DLMF 5.11.13 after shifting a up
    while big < 60:
        ratio *= big / (big + 0.5)
        big += 1.0
    t = 1.0 / big
    ratio *= math.sqrt(big) * (1 - t / 8 + t**2 / 128 + 5 * t**3 / 1024 - 21 * t**4 / 32768
                               - 399 * t**5 / 262144 + 869 * t**6 / 4194304)
    f = f.clamp(min=1e-10)
    z, w = df / (df + f), f / (df + f)
    front = ratio / math.sqrt(math.pi) * torch.exp(a * torch.log1p(-w)) * torch.sqrt(w)

    def cf(p, q, x):
        c, d = torch.ones_like(x), 1.0 / (1.0 - (p + q) * x / (p + 1))
        h = d.clone()
        for k in range(1, 600):
            for num in (k * (q - k) * x / ((p + 2 * k - 1) * (p + 2 * k)),
                        -(p + k) * (p + q + k) * x / ((p + 2 * k) * (p + 2 * k + 1))):
                d = 1.0 / (1.0 + num * d)
                c = 1.0 + num / c
                h = h * c * d
        return h

    direct = front * cf(a, 0.5, z.clamp(max=(a + 1) / (a + 2.5))) / a
    other = 1.0 - front * cf(0.5, a, w.clamp(max=1.5 / (a + 2.5))) / 0.5
    return torch.where(z < (a + 1) / (a + 2.5), direct, other)


def _exact_assoc(ev, U, W, y, genotypes, mode, m):
    """Statistics of every test of ``mode``, each (phi, m); ``genotypes(s, e)`` gives
    imputed SNPs.  Fields are named as in the package's per-chunk output."""
    n, phi = ev.numel(), y.shape[1]
    Wr = (U @ torch.from_numpy(W).to("cuda")).T.contiguous()
    Yr = (U @ torch.from_numpy(y).to("cuda")).T.contiguous()
    keys = eng.MODE_KEYS[mode]
    out = {k: torch.empty((phi, m), dtype=torch.float64, device="cuda") for k in keys}
    null = [_null_model(ev, Wr, Yr[f]) for f in range(phi)] if mode != 1 else []
    step = max(1, 30_000_000 // n)
    for s in range(0, m, step):
        e = min(m, s + step)
        X = genotypes(s, e) @ U.T
        for f in range(phi):
            ex = _Exact(ev, Wr, Yr[f], X)
            if mode in (1, 4):
                lam, logl, (xx, xy, yy), pyy = ex.search(True)
                tau = ex.df / pyy
                var = 1.0 / (tau * xx)
                out["lambda_remle"][f, s:e] = torch.exp(lam)
                out["logl_h1"][f, s:e] = logl
                out["beta"][f, s:e] = xy / xx
                out["se"][f, s:e] = torch.sqrt(var.abs())
                out["p_wald"][f, s:e] = _f_sf((yy - pyy) * tau, ex.df)
            if mode in (2, 4):
                lam, logl, _, _ = ex.search(False)
                out["lambda_mle"][f, s:e] = torch.exp(lam)
                out["logl_mle"][f, s:e] = logl
                stat = (2.0 * (logl - null[f][1])).clamp(min=0.0)
                out["p_lrt"][f, s:e] = torch.erfc(torch.sqrt(0.5 * stat))
            if mode in (3, 4):
                lam0 = torch.tensor([null[f][0]], dtype=torch.float64, device="cuda")
                _, (xx, xy, yy), pyy = ex.logl(torch.log(lam0), False)
                if mode == 3:
                    out["beta"][f, s:e] = xy / xx
                    out["se"][f, s:e] = torch.sqrt((pyy / (ex.df * xx)).abs())
                out["p_score"][f, s:e] = _f_sf(n * xy * xy / (yy * xx), ex.df)
    return out


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "assoc":
        if case["n"] * float(case["m"]) * case["phi"] > 4e8:  # over the time an exact pass may take
            return None
        U, evals, W, y = _cohort_inputs(case, seed)
        packed, sidx, means, _ = _records(case, seed)
        mu = torch.from_numpy(means).to("cuda")[:, None]

        def genotypes(s, e):
            # the streaming path imputes with its float32 means
            x = _imputed(packed[s:e], case["n"], sidx)
            called = (x == 0) | (x == 1) | (x == 2)
            return torch.where(called, x, mu[s:e].expand_as(x))

        return _exact_assoc(evals, U, W, y, genotypes, case["mode"], case["m"])
    if kind == "cohort":
        U, evals, W, y = _cohort_inputs(case, seed)
        Wr = (U @ torch.from_numpy(W).to("cuda")).T.contiguous()
        Yr = (U @ torch.from_numpy(y).to("cuda")).T.contiguous()
        out = {"UtW": Wr, "Uty": Yr}
        if case["mode"] != 1:
            null = np.array([_null_model(evals, Wr, Yr[f]) for f in range(case["phi"])])
            out.update(lam0=torch.from_numpy(null[:, 0].copy()), logl0=torch.from_numpy(null[:, 1].copy()))
        return out
    packed = synth.packed_records_device(case["n"], case["m"], case["missing"], seed)
    if kind == "kin_mem":
        return _kinship(packed, case["n"]).cpu().numpy()
    if kind == "kin_bed":
        return _kinship(packed, case["n"])
    state = prepare(case, seed)
    evals, vecs = torch.linalg.eigh(torch.from_numpy(state["K"]).to("cuda"))
    evals = torch.where(evals.abs() < 1e-10, torch.zeros_like(evals), evals)
    _, _, means, _ = _records(case, seed)
    mu = torch.from_numpy(means).to("cuda")[:, None]

    def genotypes(s, e):
        x = _imputed(packed[s:e], case["n"])
        called = (x == 0) | (x == 1) | (x == 2)
        return torch.where(called, x, mu[s:e].expand_as(x))

    got = _exact_assoc(evals, vecs.T.contiguous(), state["W"], state["y"][:, None], genotypes,
                       case["mode"], case["m"])
    field = {"logl_H1": "logl_h1", "l_remle": "lambda_remle", "l_mle": "lambda_mle"}
    out = {k: got[field.get(k, k)][0] for k in _RECORD[case["mode"]]}
    out["af"] = mu[:, 0] / 2
    return out
