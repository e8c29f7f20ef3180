"""F-test p-values at the edges of their two forms: the large-a expansion is taken for
df / 2 >= 25 and -log z <= 0.7, z = df / (df + F); the continued fraction elsewhere."""

import numpy as np
import pytest
import scipy.special

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [12, 51, 52, 53, 400, 3001])
def test_wald_p_values_follow_betainc_across_both_forms(n):
    import torch

    from jamma_b200 import engine as eng

    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    ev = np.sort(rng.uniform(0.1, 2.0, n))
    y = rng.standard_normal(n)
    cohort = eng.DeviceCohort(ev, q, None, y, 1)
    # SNPs correlated with y by rho: F from ~0 to far past both limits (F = df rho^2/(1-rho^2))
    rho = np.concatenate([np.linspace(0.0, 0.999, 300), [1e-3, 1e-2]])
    g = (rho[:, None] * (y - y.mean()) / y.std()
         + np.sqrt(1 - rho[:, None] ** 2) * rng.standard_normal((rho.size, n)))
    out = cohort.associate_genotypes(torch.from_numpy(np.ascontiguousarray(g)).cuda())
    beta, se, p = (out[k][0].cpu().numpy() for k in ("beta", "se", "p_wald"))
    df = n - 2.0
    f = (beta / se) ** 2
    ref = scipy.special.betainc(df / 2, 0.5, df / (df + np.maximum(f, 1e-10)))
    # F as formed on the device cancels (yy - pyy): relative error up to a few eps * df / F,
    # which moves log p by at most (df + 1) / 2 * F / (df + F) times that
    tol = 1e-13 * (1 + df) * np.maximum(1.0, f / (df + f) * df)
    ok = ref > 1e-290
    assert ok.sum() > 100
    np.testing.assert_array_less(np.abs(p[ok] / ref[ok] - 1), np.maximum(tol[ok], 1e-11))
