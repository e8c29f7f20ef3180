"""The missing-call walk of the INT8 kinship at the edges of its launch shapes: 2, 3 and 4 SNPs
per table (n up to 2044, up to 5120, above), one and two CTAs per sample (n above 10 240),
words that end inside a group of four, lists that are empty, shorter than a table and not a
multiple of one, against a float64 product over the imputed matrix."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p", [(5, 40), (63, 33), (2044, 70), (2049, 64), (5120, 37), (5121, 41),
                                 (6143, 45), (10240, 30), (10241, 35)])
def test_missing_call_walk_across_launch_shapes(n, p, monkeypatch):
    import torch

    from jamma_b200 import kinship as KM

    monkeypatch.setattr(KM, "TC_MISSING_DENSITY", 2.0)  # always the walk
    rng = np.random.default_rng(n)
    g = rng.binomial(2, rng.uniform(0.1, 0.9, p), (n, p)).astype(np.float64)
    for i, k in ((0, 0), (1, 1), (2, 2), (3, 3), (n // 2, 7), (n - 1, 9)):
        g[i, rng.permutation(p)[:k]] = np.nan
    g[n - 2, : p - 1] = np.nan  # nearly every call of a sample
    g[rng.random((n, p)) < 0.01] = np.nan
    g[0] = np.nan_to_num(g[0], nan=1.0)  # a sample without missing calls
    got = KM.compute_centered_kinship(g, precision="int8")
    x = torch.from_numpy(np.where(np.isnan(g), np.nanmean(g, 0), g) - np.nanmean(g, 0)).cuda()
    keep = torch.from_numpy(np.nanvar(g, 0) > 0).cuda()
    x = x[:, keep]
    ref = (x @ x.T / x.shape[1]).cpu().numpy()
    # a few roundings of sums of p terms of size <= 4, divided by p
    assert np.abs(got - ref).max() <= 64 * p * 2.0 ** -53 * 4 / p * 4
