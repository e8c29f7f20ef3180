"""FP64 centered kinship through the exact integer Gram of the shifted calls, against extended
precision and against the FP64 product (src/jamma/kinship/compute.py:46-57)."""

import numpy as np
import pytest
import torch

from jamma_b200 import kinship as kk

U = 2.0 ** -53


def _calls(n, p, miss, seed):
    rng = np.random.default_rng(seed)
    c = rng.binomial(2, rng.uniform(0.02, 0.98, p)[:, None], (p, n)).astype(np.int8)
    c[rng.random((p, n)) < miss] = 3
    if p > 3:
        c[0, : n // 2], c[0, n // 2:] = 0, 1  # mean 1/2 (n even): rounds to even
        c[1, : n // 2], c[1, n // 2:] = 1, 2  # mean 3/2
        c[2] = 3                              # no call at all
        c[3] = 2                              # constant: zero terms
    obs = (c != 3).sum(1)
    mu = np.where(c == 3, 0, c).sum(1) / np.maximum(obs, 1)
    return c, mu


@pytest.mark.gpu
@pytest.mark.parametrize("n,p,miss,block,chunk", [
    (1, 5, 0.0, 65536, 16384),
    (31, 1, 0.0, 65536, 16384),
    (32, 257, 0.05, 65536, 16384),
    (130, 700, 0.02, 300, 128),     # three Grams, chunks cut at the blocks' ends
    (258, 129, 0.3, 64, 16384),
    (1026, 515, 0.01, 256, 100),
    (2050, 300, 0.02, 65536, 16384),  # three SNPs per table
    (5130, 130, 0.02, 128, 16384),    # four SNPs per table, two words per thread
])
def test_exact_form_against_extended_precision(n, p, miss, block, chunk, monkeypatch):
    monkeypatch.setattr(kk._KinshipExact, "BLOCK", block)
    monkeypatch.setattr(kk._KinshipExact, "MAX_CHUNK", chunk)
    c, mu = _calls(n, p, miss, n + p)
    ld = (n + 15) // 16 * 16 + (1 if n == 258 else 0)  # an odd stride: the scalar paths
    codes = torch.zeros((p, ld), dtype=torch.int8, device="cuda")
    codes[:, :n] = torch.from_numpy(c).cuda()
    has_missing = bool((c == 3).any())
    acc = kk._KinshipExact(n, p, has_missing)
    cut = p // 3 + 1
    mu_d = torch.from_numpy(mu).cuda()
    for s in range(0, p, cut):
        acc.add(codes[s:s + cut], mu[s:s + cut], mu_d[s:s + cut], has_missing)
    K = acc.finish().cpu().numpy()
    assert np.array_equal(K, K.T)
    rows = np.unique(np.linspace(0, n - 1, min(n, 40)).astype(int))
    X = np.where(c == 3, 0, c.astype(np.longdouble) - mu.astype(np.longdouble)[:, None])[:, rows]
    ref = X.T @ X  # p K
    # Q's entries are sums of at most L terms of size <= 1, each addition rounded once, b of at
    # most L terms of 1/4; the other terms are exact in two doubles and K is rounded once
    L = (c[:, rows] == 3).sum(0)
    L2 = L[:, None] + L[None, :] + 8.0
    tol = U * (4 * np.abs(ref) + 2 * L2 * L2 * (1.0 if has_missing else 0.0)) + 1e-26 * p * p
    err = np.abs(K[np.ix_(rows, rows)].astype(np.longdouble) * p - ref)
    assert np.all(err <= tol), float((err / tol).max())


@pytest.mark.gpu
@pytest.mark.parametrize("n,p,miss", [(1001, 10007, 0.01), (1204, 9000, 0.0)])
def test_public_call_takes_the_exact_form_and_agrees_with_the_product(n, p, miss, monkeypatch):
    c, _ = _calls(n, p, miss, 7)
    g = np.where(c == 3, np.nan, c.astype(np.float64)).T
    used = []
    real = kk._KinshipExact.finish
    monkeypatch.setattr(kk._KinshipExact, "finish", lambda self: used.append(1) or real(self))
    K = kk.compute_centered_kinship(g)
    assert used
    monkeypatch.setattr(kk, "exact_form_pays", lambda *a: False)
    P = kk.compute_centered_kinship(g)
    assert len(used) == 1
    # the product adds p terms of size <= 4 in FP64
    assert np.max(np.abs(K - P)) <= 4 * p * U * np.max(np.abs(P))


def test_rule_edges():
    assert kk.exact_form_pays(1000, 10000, 0)
    assert not kk.exact_form_pays(999, 20000, 0)
    assert not kk.exact_form_pays(1000, 9999, 0)
    assert not kk.exact_form_pays(20000, 999, 0)
    assert not kk.exact_form_pays(65537, 10000, 0)
    assert not kk.exact_form_pays(2000, 10000, 2000 * 10000 // 20)
    assert kk.exact_form_pays(8000, 10000, 8000 * 10000 // 20)
    assert not kk.exact_form_pays(8000, 10000, 8000 * 10000 // 5)
