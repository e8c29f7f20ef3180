"""The FP64 rotation of genotype calls from exact INT8 digit planes, against 80-bit sums, at
the edges of its tiles: 32 eigenvectors x 64 SNPs with missing calls (128 without), K slices
of 128 samples, unaligned code rows, and the calls an imputation mean does and does not touch."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U64 = 2.0 ** -53


@pytest.mark.parametrize("n,m,pad,missing", [
    (3, 1, 0, 0.3), (31, 63, 1, 0.1), (32, 64, 0, 0.1), (33, 65, 5, 0.1), (127, 129, 0, 0.02),
    (128, 128, 0, 0.0), (129, 127, 15, 0.0), (500, 70, 12, 0.01), (700, 257, 4, 0.0), (1030, 300, 2, 0.6)])
def test_rotation_of_calls_is_exact_to_rounding(n, m, pad, missing):
    import torch

    from jamma_b200 import _native
    from jamma_b200 import engine as eng
    from jamma_b200.device import ptr, stream_handle, workspace

    rng = np.random.default_rng(n * 1000 + m)
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    q[:, -1] *= 1e-8      # eigenvectors of other scales: each has its own
    if n > 40:
        q[:, 7] = 0.0
        q[:, 8] *= 2.0 ** 40
    z = rng.integers(0, 3, (m, n)).astype(np.int8)
    miss = rng.random((m, n)) < missing
    if missing:
        miss[0, 0] = True
    codes = np.zeros((m, n + pad), dtype=np.int8)
    codes[:, :n] = np.where(miss, 3, z)
    mu = rng.uniform(0, 2, m)
    if missing:
        mu[~miss.any(1)] = np.nan  # not used: no call of the SNP is missing
    # columns of U are the rows of the device tensor
    ut = torch.from_numpy(np.ascontiguousarray(q.T)).cuda()
    dc, dm = torch.from_numpy(codes).cuda(), torch.from_numpy(mu).cuda()
    planes = eng.exact_split(ut)
    lib = _native.load()
    ws = workspace(lib.jb_rotate_codes_f64_workspace_size(n, m))
    lz = np.where(miss, 0, z).astype(np.longdouble)
    qz = lz @ q.astype(np.longdouble)
    qm = miss.astype(np.longdouble) @ q.astype(np.longdouble)
    mz = np.where(miss.any(1), mu, 0.0)[:, None]
    exact = qz + mz * qm
    # the dropped remainder (2.93e-17 of max|U_col| per unit of |g|) and a few roundings of the
    # sums' own size: six Horner steps, the imputation's multiply-add and the scale
    g1 = (lz.sum(1) + mz[:, 0] * miss.sum(1))[:, None]
    bound = 3e-17 * np.abs(q).max(0)[None, :] * g1 + 10 * U64 * (np.abs(qz) + mz * np.abs(qm))
    for has_missing in ((1,) if missing else (1, 0)):
        x = torch.full((m, n), -7.0, dtype=torch.float64, device="cuda")
        _native.call("jb_rotate_codes_f64", ptr(planes), n, ptr(dc), n + pad, m, ptr(dm), has_missing,
                     ptr(x), n, ptr(ws), ws.numel(), stream_handle())
        err = np.abs(x.cpu().numpy().astype(np.longdouble) - exact)
        assert np.all(err <= bound), (has_missing, float((err / np.maximum(bound, 1e-300)).max()))
        assert int(ws[:4].view(torch.int32)[0]) == 0
    if missing and (n + pad) % 16 == 0:  # the promise of no missing calls is checked
        x.fill_(0)
        _native.call("jb_rotate_codes_f64", ptr(planes), n, ptr(dc), n + pad, m, ptr(dm), 0, ptr(x), n,
                     ptr(ws), ws.numel(), stream_handle())
        assert np.all(np.abs(x.cpu().numpy().astype(np.longdouble) - exact) <= bound)
    # no further off than the FP64 GEMM of the imputed calls
    if n >= 127:
        g = torch.from_numpy(np.where(miss, np.nan_to_num(mu)[:, None], z).astype(np.float64)).cuda()
        gemm = np.abs(eng.rotate(ut, g).cpu().numpy().astype(np.longdouble) - exact)
        assert np.linalg.norm(err.astype(float)) <= np.linalg.norm(gemm.astype(float))


def test_non_finite_eigenvectors_give_nan():
    import torch

    from jamma_b200 import engine as eng

    n = 64
    u = np.linalg.qr(np.random.default_rng(0).standard_normal((n, n)))[0]
    u[3, 5] = np.nan
    ut = torch.from_numpy(np.ascontiguousarray(u.T)).cuda()
    coh = eng.DeviceCohort.__new__(eng.DeviceCohort)
    coh.n, coh.ozaki, coh._rot_ws = n, eng.exact_split(ut), None
    x = coh.rotate_codes_f64(torch.ones((4, 64), dtype=torch.int8, device="cuda"),
                             torch.ones(4, dtype=torch.float64, device="cuda")).cpu().numpy()
    assert np.isnan(x[:, 5]).all() and np.isfinite(np.delete(x, 5, 1)).all()
