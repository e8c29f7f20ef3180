"""Centered (GEMMA -gk 1) and standardized (-gk 2) kinship on the GPU.

``compute_centered_kinship`` keeps jamma's signature and semantics
(src/jamma/kinship/compute.py:93-226): SNPs are filtered by MAF / missing rate /
monomorphism with statistics in the input dtype, each kept SNP is mean-imputed and
centred with its float64 mean over observed samples, and K = Xc Xc^T / p_kept.
Genotypes travel to the device as packed 2-bit records and are decoded there.
"""

from __future__ import annotations

import numpy as np
import torch

from jamma_b200 import _native
from jamma_b200.device import empty, ptr, require_cuda, stream_handle, workspace
from jamma_b200.engine import decode_packed, pack_on_device, pass1_counts
from jamma_b200.io import BedFile, apply_snp_list_mask, open_bed


def snp_stats_from_counts(counts: np.ndarray, n: int, dtype=np.float32):
    """(mean, miss, polymorphic) from device counts {n_obs, sum, n_het, n_hom2}.

    The mean is NumPy's ``nanmean`` in ``dtype``: the integer sum divided by the count
    in float64, then stored in ``dtype`` (0 for all-missing SNPs).  ``polymorphic`` is
    ``nanvar > 0``: at least two different observed genotypes.
    """
    n_obs = counts[:, 0].astype(np.int64)
    s = counts[:, 1].astype(np.float64)
    het = counts[:, 2].astype(np.int64)
    hom2 = counts[:, 3].astype(np.int64)
    hom0 = n_obs - het - hom2
    with np.errstate(invalid="ignore", divide="ignore"):
        mean = np.where(n_obs > 0, s / np.maximum(n_obs, 1), 0.0).astype(dtype)
    poly = ((hom0 > 0).astype(int) + (het > 0) + (hom2 > 0)) >= 2
    return mean, (n - n_obs).astype(np.int64), poly


def snp_sd_from_counts(counts: np.ndarray, n: int) -> np.ndarray:
    """Per-SNP standard deviation of the mean-imputed genotypes over all n samples, as
    ``impute_center_and_standardize`` forms it (src/jamma/kinship/missing.py:102-108):
    var = mean(x_imputed^2) - mean^2 with the float64 mean over observed samples."""
    n_obs = counts[:, 0].astype(np.float64)
    s = counts[:, 1].astype(np.float64)
    sq = counts[:, 2].astype(np.float64) + 4.0 * counts[:, 3].astype(np.float64)
    mu = np.where(n_obs > 0, s / np.maximum(n_obs, 1), 0.0)
    var = (sq + (n - n_obs) * mu * mu) / n - mu * mu
    return np.sqrt(np.maximum(var, 0.0))


def filter_mask(mean, miss, poly, n, maf_threshold, miss_threshold):
    """``compute_snp_filter_mask`` (src/jamma/core/snp_filter.py:59-91)."""
    af = np.asarray(mean, dtype=np.float64) / 2.0
    maf = np.minimum(af, 1.0 - af)
    keep = (maf >= maf_threshold) & ((miss / n) <= miss_threshold) & poly
    return keep, af


class _KinshipAccumulator:
    """FP64 centered (or, given per-SNP sd, standardized) Gram accumulated over SNP
    batches (``_accumulate_kinship``)."""

    def __init__(self, n: int, batch: int):
        self.n, self.batch = n, batch
        self.K = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        self.ws = workspace(_native.load().jb_kinship_f64_workspace_size(n, batch))
        self.p = 0

    def add(self, codes: torch.Tensor, means64: torch.Tensor, sd64: torch.Tensor | None = None) -> None:
        m, ld = codes.shape
        for s in range(0, m, self.batch):
            e = min(s + self.batch, m)
            if sd64 is None:
                _native.call("jb_kinship_accumulate_f64", ptr(codes[s:e]), ld, self.n, e - s,
                             ptr(means64[s:e]), ptr(self.K), self.n, ptr(self.ws), self.ws.numel(),
                             stream_handle())
            else:
                _native.call("jb_kinship_accumulate_std_f64", ptr(codes[s:e]), ld, self.n, e - s,
                             ptr(means64[s:e]), ptr(sd64[s:e]), ptr(self.K), self.n, ptr(self.ws),
                             self.ws.numel(), stream_handle())
        self.p += m

    def finish(self) -> torch.Tensor:
        _native.call("jb_kinship_finalize", ptr(self.K), self.n, self.n, 1.0 / self.p,
                     stream_handle())
        return self.K


class _KinshipExact:
    """The FP64 centered kinship through the exact INT8 tensor-core Gram of the calls less
    rint(mean), with the centring terms in sums of two doubles (jb_kinship_exact_*): nothing
    but the missing-call terms and the last division rounds, so that K is at least as close to
    exact sums as the accumulated FP64 product.  SNPs fill blocks of BLOCK operand columns;
    each full block is one Gram added to the int32 sums (at most 4 per SNP)."""

    MAX_CHUNK = 16384
    BLOCK = 65536

    def __init__(self, n: int, p_kept: int, has_missing: bool, chunk: int = MAX_CHUNK):
        """``chunk``: most SNPs that one call of :meth:`add` brings."""
        self.n, self.p = n, p_kept
        self.cols = min(self.BLOCK, p_kept)
        self.ldz = (self.cols + 127) // 128 * 128
        self.Zs = torch.empty((n, self.ldz), dtype=torch.int8, device="cuda")
        self.C = torch.empty((n, n), dtype=torch.int32, device="cuda")
        self.vec = torch.zeros((3, n), dtype=torch.float64, device="cuda")  # a, a_lo, b
        self.Q = (torch.zeros if has_missing else torch.empty)(
            (n, n), dtype=torch.float64, device="cuda")
        self.has_missing = has_missing
        lib = _native.load()
        self.step = min(self.MAX_CHUNK, self.cols, chunk)
        self.ws = workspace(lib.jb_kinship_exact_workspace_size(n, self.step))
        self.gram_ws = workspace(lib.jb_gram_i8_workspace_size(n))
        self._status: list[torch.Tensor] = []
        self.col, self.blocks = 0, 0
        self.sum_sq = np.longdouble(0.0)

    @staticmethod
    def device_bytes(n: int, p_kept: int) -> int:
        lib = _native.load()
        cols = min(_KinshipExact.BLOCK, p_kept)
        return (12 * n * n + n * (cols + 128) + lib.jb_gram_i8_workspace_size(n)
                + lib.jb_kinship_exact_workspace_size(n, min(_KinshipExact.MAX_CHUNK, cols)))

    def add(self, codes: torch.Tensor, mu64_host: np.ndarray, mu: torch.Tensor,
            has_missing: bool) -> None:
        """Add a chunk of decoded codes (m, ld) with its means on the host and the device."""
        m, ld = codes.shape
        d = (mu64_host - np.rint(mu64_host)).astype(np.longdouble)
        self.sum_sq += np.sum(d * d)
        st, s = stream_handle(), 0
        while s < m:
            e = s + min(m - s, self.step, self.cols - self.col)
            _native.call("jb_kinship_exact_accumulate", ptr(codes[s:e]), ld, self.n, e - s, ptr(mu[s:e]),
                         int(has_missing), ptr(self.Zs), self.ldz, self.col, ptr(self.vec[0]),
                         ptr(self.vec[1]), ptr(self.vec[2]), ptr(self.Q), self.n, ptr(self.ws),
                         self.ws.numel(), st)
            self.col += e - s
            if self.col == self.cols:
                self._gram()
            s = e

    def _gram(self) -> None:
        entry = "jb_gram_i8_add" if self.blocks else "jb_gram_i8"
        _native.call(entry, ptr(self.Zs), self.n, self.col, self.ldz, ptr(self.C), self.n,
                     ptr(self.gram_ws), self.gram_ws.numel(), stream_handle())
        self._status.append(self.gram_ws[:4].clone())
        self.blocks += 1
        self.col = 0

    def finish(self) -> torch.Tensor:
        if self.col:
            self._gram()
        hi = float(self.sum_sq)
        _native.call("jb_kinship_exact_finalize", ptr(self.C), self.n, self.n, ptr(self.vec[0]),
                     ptr(self.vec[1]), ptr(self.vec[2]), hi, float(self.sum_sq - np.longdouble(hi)),
                     ptr(self.Q) if self.has_missing else None, self.n, self.p, ptr(self.Q), self.n,
                     stream_handle())
        status = torch.cat(self._status).view(torch.int32).cpu().numpy()
        if np.any(status != 0):
            raise RuntimeError(f"INT8 Gram pipeline reported status {status[status != 0][0]}")
        return self.Q


# Where the exact form is the faster one.  It pays ~0.25 ms of launches, the n^2 passes of its
# int32 and missing-call sums, and a walk over the missing calls; the product runs at the FP64
# rate.  Measured, product against exact form in ms at 0 / 1 / 5 / 10 % missing calls:
#   n = 400,    p = 20 000   0.47 : 0.52 / 0.68 / 0.97 / 1.3
#   n = 1200,   p =  5000    0.43 : 0.28 / 0.37 / 0.57 / 0.81
#   n = 1940,   p = 12 226   1.70 : 0.42 / 0.71 / 1.4  / 2.4
#   n = 4001,   p = 20 000   10.1 : 0.95 / 1.8  / 3.8  / 6.3
#   n = 20 000, p = 30 011   340  : 7.5  / 34   / 121  / 228
# The lines lie on the safe side of the table: n = 1200, p = 5000 (7.2e9) still takes the product,
# 0.06 to 0.15 ms more with up to 1 % missing.
# The memory limit leaves half of what is free to the caller: the exact form holds 12 n^2 bytes
# and the operand block where the product holds 8 n^2.
EXACT_MIN_WORK = 1.0e10       # n^2 p
EXACT_MIN_SAMPLES = 1000
EXACT_MAX_SAMPLES = 65536
EXACT_MIN_SNPS = 1000         # below, the n^2 passes weigh more than the product
EXACT_MISSING_DENSITY = 0.03  # of all calls
EXACT_MISSING_DENSITY_WIDE = 0.1  # from EXACT_WIDE_SAMPLES samples on
EXACT_WIDE_SAMPLES = 4000


def exact_form_pays(n: int, p_kept: int, n_missing: int) -> bool:
    """Whether the FP64 centered kinship of n samples and p_kept SNPs takes the exact form."""
    density = EXACT_MISSING_DENSITY_WIDE if n >= EXACT_WIDE_SAMPLES else EXACT_MISSING_DENSITY
    return (EXACT_MIN_SAMPLES <= n <= EXACT_MAX_SAMPLES and EXACT_MIN_SNPS <= p_kept < 1 << 29
            and float(n) * n * p_kept >= EXACT_MIN_WORK and n_missing <= density * n * p_kept)


def _fp64_accumulator(n: int, p_kept: int, n_missing: int, batch: int,
                      chunk: int = _KinshipExact.MAX_CHUNK):
    """Accumulator of the FP64 centered kinship: exact form (SNPs added ``chunk`` at a time at
    most) or FP64 product."""
    if exact_form_pays(n, p_kept, n_missing):
        free = (torch.cuda.mem_get_info()[0] + torch.cuda.memory_reserved()
                - torch.cuda.memory_allocated())
        if _KinshipExact.device_bytes(n, p_kept) <= free // 2:
            return _KinshipExact(n, p_kept, n_missing > 0, chunk)
    return _KinshipAccumulator(n, batch)


# Missing-call density (fraction of a chunk's calls) above which the correction terms run on the
# INT8 tensor cores instead of the FP64 walk over each sample's missing SNPs.  The tensor-core
# form walks the same lists for its missing x missing term, so its dense product only replaces
# the building of the walk's wider tables: ms per chunk, walk : tensor cores, at 3 / 12 / 20 /
# 30 % missing: n = 20 000, 16 384 SNPs 32 : 49, 116 : 122, 192 : 187, 286 : 269; n = 1940,
# 12 226 SNPs 0.80 : 1.12, 2.5 : 2.7, 4.0 : 4.1, 5.8 : 5.9.
TC_MISSING_DENSITY = 0.2


class _KinshipI8:
    """Exact INT8 tensor-core Gram + FP64 centring / missing-call corrections.

    MAX_CHUNK: SNPs per correction call (longer chunks are split).

    SNP chunks are transposed into the sample-major int8 operand (missing -> 0) and
    their correction vectors accumulated; ``finish`` runs the tcgen05 Gram once over all
    kept SNPs and combines the terms (see jb_gram.cu for the identity used).
    """

    MAX_CHUNK = 16384

    def __init__(self, n: int, p_kept: int):
        self.n, self.p = n, p_kept
        self.ldz = (p_kept + 127) // 128 * 128
        self.Zs = torch.zeros((n, self.ldz), dtype=torch.int8, device="cuda")
        self.a = torch.zeros(n, dtype=torch.float64, device="cuda")
        self.b = torch.zeros(n, dtype=torch.float64, device="cuda")
        self.RT = None
        self.sum_mu2 = 0.0
        self.col = 0
        self._status: list[torch.Tensor] = []
        self._density_scale = 1.0

    def add(self, codes: torch.Tensor, mu64: torch.Tensor, has_missing: bool,
            n_missing: int | None = None) -> None:
        """Add a chunk of decoded codes (m, ld).  ``n_missing``: the chunk's number of
        missing calls (from pass-1 counts; counted on the device when not given); chunks
        whose missing calls exceed TC_MISSING_DENSITY take the tensor-core correction."""
        m, ld = codes.shape
        if has_missing and n_missing is None:
            n_missing = int((codes[:, : self.n] == 3).sum())
        if m > self.MAX_CHUNK:  # the correction kernels take at most MAX_CHUNK SNPs per call
            for s in range(0, m, self.MAX_CHUNK):
                e = min(s + self.MAX_CHUNK, m)
                # the density test uses the whole chunk's average
                self._density_scale = m / (e - s)
                self.add(codes[s:e], mu64[s:e], has_missing, n_missing)
            self._density_scale = 1.0
            return
        st = stream_handle()
        if has_missing and self.RT is None:
            self.RT = torch.zeros((self.n, self.n), dtype=torch.float64, device="cuda")
        _native.call("jb_codes_to_sample_major", ptr(codes), ld, self.n, m, ptr(self.Zs), self.ldz,
                     self.col, None, 0, st)
        lib = _native.load()
        if has_missing and self.col % 16 == 0 and \
                n_missing > TC_MISSING_DENSITY * self.n * m * self._density_scale:
            ws = workspace(lib.jb_kinship_i8_tc_workspace_size(self.n, m))
            _native.call("jb_kinship_i8_corrections_tc", ptr(codes), ld, ptr(self.Zs), self.ldz,
                         self.col, self.n, m, ptr(mu64), ptr(self.a), ptr(self.b),
                         ptr(self.RT), self.n, ptr(ws), ws.numel(), st)
        else:
            ws = workspace(lib.jb_kinship_i8_corrections_workspace_size(self.n, m))
            _native.call("jb_kinship_i8_corrections", ptr(codes), ld, int(has_missing), self.n, m,
                         ptr(mu64), ptr(self.a), ptr(self.b), ptr(self.RT), self.n, ptr(ws),
                         ws.numel(), st)
        if has_missing:
            self._status.append(ws[:4].clone())  # status word, checked in finish()
        self.col += m

    def add_sum_mu2(self, mu64_host: np.ndarray) -> None:
        self.sum_mu2 += float(np.sum(np.asarray(mu64_host, dtype=np.float64) ** 2))

    def gram(self) -> torch.Tensor:
        """Exact int32 Gram of the accumulated calls (upper triangle, column-major)."""
        n = self.n
        st = stream_handle()
        C = torch.empty((n, n), dtype=torch.int32, device="cuda")
        ws = workspace(_native.load().jb_gram_i8_workspace_size(n))
        _native.call("jb_gram_i8", ptr(self.Zs), n, self.p, self.ldz, ptr(C), n, ptr(ws), ws.numel(), st)
        status = np.zeros(1, dtype=np.int32)
        _native.call("jb_gram_status", ptr(ws), status.ctypes.data, st)
        if status[0] != 0:
            raise RuntimeError(f"INT8 Gram pipeline reported status {int(status[0])}")
        self.Zs = None  # the operand is no longer needed
        return C

    def finish(self) -> torch.Tensor:
        n = self.n
        if self._status:
            st = torch.cat(self._status).view(torch.int32).cpu().numpy()
            if np.any(st != 0):
                raise RuntimeError(f"tensor-core kinship correction reported status {st[st != 0][0]}")
        C = self.gram()
        K = torch.empty((n, n), dtype=torch.float64, device="cuda")
        _native.call("jb_kinship_i8_finalize", ptr(C), n, n, ptr(self.a), ptr(self.b), self.sum_mu2,
                     ptr(self.RT), n, self.p, ptr(K), n, stream_handle())
        return K


def _kinship_from_packed(packed_dev: torch.Tensor, n: int, batch_size: int, maf_threshold: float,
                         miss_threshold: float, stat_dtype, precision: str = "fp64",
                         standardized: bool = False) -> tuple[torch.Tensor, int]:
    codes, counts = decode_packed(packed_dev, n, None, n, (n + 15) // 16 * 16)
    mean, miss, poly = snp_stats_from_counts(counts.cpu().numpy(), n, stat_dtype)
    keep, _ = filter_mask(mean, miss, poly, n, maf_threshold, miss_threshold)
    idx = np.where(keep)[0]
    if idx.size == 0:
        raise ValueError(
            f"No SNPs passed filtering (maf>={maf_threshold}, miss<={miss_threshold}, "
            f"polymorphic). Original SNP count: {packed_dev.shape[0]}"
        )
    c = counts.cpu().numpy()[idx]
    mu64 = torch.from_numpy(c[:, 1] / np.maximum(c[:, 0], 1)).to("cuda")  # float64 nanmean
    sel = torch.from_numpy(idx).to("cuda")
    if standardized:
        acc = _KinshipAccumulator(n, max(1, min(batch_size, 8192)))
        acc.add(codes.index_select(0, sel), mu64, torch.from_numpy(snp_sd_from_counts(c, n)).to("cuda"))
        return acc.finish(), idx.size
    if precision == "int8":
        acc = _KinshipI8(n, idx.size)
        acc.add(codes.index_select(0, sel), mu64, bool(np.any(c[:, 0] < n)),
                n_missing=int((n - c[:, 0]).sum()))
        acc.add_sum_mu2(c[:, 1] / np.maximum(c[:, 0], 1))
        return acc.finish(), idx.size
    n_missing = int((n - c[:, 0]).sum())
    acc = _fp64_accumulator(n, idx.size, n_missing, max(1, min(batch_size, 8192)))
    if isinstance(acc, _KinshipExact):
        acc.add(codes.index_select(0, sel), c[:, 1] / np.maximum(c[:, 0], 1), mu64, n_missing > 0)
    else:
        acc.add(codes.index_select(0, sel), mu64)
    return acc.finish(), idx.size


def _resident_records(bed: BedFile, n: int, int8: bool) -> torch.Tensor | None:
    """Device buffer for all records of the file, or None when they would take more than a
    quarter of the memory that the accumulation over n samples leaves free."""
    free = (torch.cuda.mem_get_info()[0] + torch.cuda.memory_reserved()
            - torch.cuda.memory_allocated())
    # n x n: int32 Gram, missing-call terms and result; per SNP: the whole INT8 operand, or the
    # chunk buffers of either form
    need = 20 * n * n + n * (bed.n_snps if int8 else 65536) + 10 * n * 16384
    if bed.n_snps * bed.bytes_per_snp > (free - need) // 4:
        return None
    return torch.empty((bed.n_snps, bed.bytes_per_snp), dtype=torch.uint8, device="cuda")


# compute_kinship_from_bed: the default chunk_size, and the chunk it and larger ones stand for on
# the device: the missing-call walk reads and writes its n^2 sums once per chunk (30 011 SNPs at
# n = 20 000 in chunks of 10 000 or 16 384: 23.3 or 20.7 ms), and two full batches of the
# FP64 product fit.  Smaller ones are a caller's limit on the chunk's buffers and are kept.
KINSHIP_CHUNK, KINSHIP_DEVICE_CHUNK = 10_000, 16_384


def _device_chunk(chunk_size: int) -> int:
    return chunk_size if chunk_size < KINSHIP_CHUNK else max(chunk_size, KINSHIP_DEVICE_CHUNK)


def _selected_records(bed: BedFile, idx: np.ndarray, step: int, kept: torch.Tensor | None):
    """Yield the records of SNPs ``idx`` on the device, ``step`` at a time: from the records that
    pass 1 left there, else read again through two pinned buffers."""
    pin = [None, None]
    done = [None, None]
    for ci, s in enumerate(range(0, idx.size, step)):
        sub = idx[s:s + step]
        if kept is not None:
            if sub[-1] - sub[0] + 1 == sub.size:  # idx increases
                yield kept[int(sub[0]):int(sub[-1]) + 1]
            else:
                yield kept.index_select(0, torch.from_numpy(sub).to("cuda"))
            continue
        b = ci % 2
        if pin[b] is None:
            pin[b] = torch.empty((min(step, idx.size), bed.bytes_per_snp), dtype=torch.uint8,
                                 pin_memory=True)
        if done[b] is not None:
            done[b].synchronize()
        bed.take_into(sub, pin[b].numpy()[: sub.size])
        rec = pin[b][: sub.size].to("cuda", non_blocking=True)
        done[b] = torch.cuda.Event()
        done[b].record()
        yield rec


def compute_standardized_kinship(genotypes: np.ndarray, batch_size: int = 10000,
                                 maf_threshold: float = 0.0, miss_threshold: float = 1.0,
                                 check_memory: bool = True) -> np.ndarray:
    """GEMMA -gk 2 relatedness matrix of an in-memory (n, p) genotype matrix.

    Keeps ``compute_standardized_kinship``'s signature and semantics
    (src/jamma/kinship/compute.py:229-360): the same SNP filter as -gk 1, then each kept
    SNP is mean-imputed, centred and divided by its standard deviation over all samples
    (``impute_center_and_standardize``, src/jamma/kinship/missing.py:64-119), and
    K = Z Z^T / p_kept.  FP64 on the device (per-SNP weights do not fit an exact integer
    Gram).
    """
    require_cuda()
    g = np.asarray(genotypes)
    n = g.shape[0]
    stat_dtype = np.float32 if g.dtype == np.float32 else np.float64
    packed = pack_on_device(g)
    K, _ = _kinship_from_packed(packed, n, batch_size, maf_threshold, miss_threshold, stat_dtype,
                                "fp64", standardized=True)
    return K.cpu().numpy()


def compute_centered_kinship(genotypes: np.ndarray, batch_size: int = 10000,
                             maf_threshold: float = 0.0, miss_threshold: float = 1.0,
                             check_memory: bool = True, precision: str = "fp64") -> np.ndarray:
    """GEMMA -gk 1 relatedness matrix of an in-memory (n, p) genotype matrix.

    ``precision="fp64"`` forms the centred Gram to FP64 accuracy: through the exact integer
    Gram of the shifted calls where ``exact_form_pays``, else as an FP64 product (cuBLAS DSYRK);
    ``precision="int8"`` runs the exact INT8 tensor-core Gram with FP64 corrections.
    """
    if precision not in ("fp64", "int8"):
        raise ValueError("precision must be 'fp64' or 'int8'")
    require_cuda()
    g = np.asarray(genotypes)
    n = g.shape[0]
    stat_dtype = np.float32 if g.dtype == np.float32 else np.float64
    packed = pack_on_device(g)
    K, _ = _kinship_from_packed(packed, n, batch_size, maf_threshold, miss_threshold, stat_dtype,
                                precision)
    return K.cpu().numpy()


def compute_kinship_from_bed(bfile, maf_threshold: float = 0.0, miss_threshold: float = 1.0,
                             chunk_size: int = KINSHIP_CHUNK, sample_idx: np.ndarray | None = None,
                             as_device: bool = False, precision: str = "fp64",
                             kinship_mode: int = 1, ksnps_indices: np.ndarray | None = None):
    """Kinship streamed from a .bed file (``compute_kinship_streaming``,
    src/jamma/kinship/compute.py:502-690): pass 1 statistics, pass 2 accumulation,
    both decoded on the device.  Pass-1 means are float32 as in jamma's streaming path.

    ``kinship_mode`` 1 = centered (-gk 1), 2 = standardized (-gk 2, FP64 only);
    ``ksnps_indices`` restricts the kinship to those SNP columns (-ksnps).
    """
    if kinship_mode not in (1, 2):
        raise ValueError(f"invalid kinship mode {kinship_mode}; use 1 or 2")
    if kinship_mode == 2 and precision != "fp64":
        raise ValueError("standardized kinship (-gk 2) is computed in FP64 only")
    if chunk_size < 1:
        raise ValueError("chunk_size must be positive")
    require_cuda()
    bed, check = open_bed(bfile)
    try:
        acc = _accumulate_from_bed(bed, maf_threshold, miss_threshold, chunk_size, sample_idx,
                                   precision, kinship_mode, ksnps_indices)
    except Exception:
        check()
        raise
    check()  # the device is still busy with the accumulation
    K = acc.finish()
    return K if as_device else K.cpu().numpy()


def _accumulate_from_bed(bed: BedFile, maf_threshold, miss_threshold, chunk_size, sample_idx,
                         precision, kinship_mode, ksnps_indices):
    """Both passes over the file; the accumulator, its last launches still running."""
    n = bed.n_samples if sample_idx is None else len(sample_idx)
    sidx = None if sample_idx is None else torch.from_numpy(
        np.asarray(sample_idx, dtype=np.int32)).to("cuda")
    kept = _resident_records(bed, n, precision == "int8")
    counts = pass1_counts(bed, sidx, n, max(chunk_size, 16384), kept)
    mean, miss, poly = snp_stats_from_counts(counts, n, np.float32)
    keep, _ = filter_mask(mean, miss, poly, n, maf_threshold, miss_threshold)
    if ksnps_indices is not None:
        apply_snp_list_mask(keep, ksnps_indices, keep.size, "Kinship SNP list")
    idx = np.where(keep)[0]
    if idx.size == 0:
        raise ValueError("No SNPs passed filtering")
    i8 = precision == "int8"
    step = _device_chunk(chunk_size)
    if i8:
        acc = _KinshipI8(n, idx.size)
    elif kinship_mode == 2:
        acc = _KinshipAccumulator(n, min(chunk_size, 8192))
    else:
        acc = _fp64_accumulator(n, idx.size, int((n - counts[idx, 0]).sum()), min(chunk_size, 8192),
                                step)
    exact = isinstance(acc, _KinshipExact)
    c = counts[idx]
    mu_host = c[:, 1] / np.maximum(c[:, 0], 1)
    mu_dev = torch.from_numpy(mu_host).to("cuda")
    sd_dev = torch.from_numpy(snp_sd_from_counts(c, n)).to("cuda") if kinship_mode == 2 else None
    s = 0
    for rec in _selected_records(bed, idx, step, kept):
        codes, _ = decode_packed(rec, bed.n_samples, sidx, n, (n + 15) // 16 * 16)
        e = s + rec.shape[0]
        n_missing = int((n - c[s:e, 0]).sum())
        if i8:
            acc.add(codes, mu_dev[s:e], n_missing > 0, n_missing=n_missing)
            acc.add_sum_mu2(mu_host[s:e])
        elif kinship_mode == 2:
            acc.add(codes, mu_dev[s:e], sd_dev[s:e])
        elif exact:
            acc.add(codes, mu_host[s:e], mu_dev[s:e], n_missing > 0)
        else:
            acc.add(codes, mu_dev[s:e])
        s = e
    return acc
