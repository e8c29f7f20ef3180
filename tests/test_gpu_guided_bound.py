"""The FP64 form's guided search against the search of direct evaluations (precision 0) where
sums cancel or shrink: a centred kinship, whose zero eigenvalue holds the intercept (its weight
stays 1 at every lambda while the other sums shrink to 1e-5), heritabilities up to 1, rare
alleles, associated SNPs, and phenotypes and covariates far from zero."""

import numpy as np
import pytest
from test_gpu_guided_search import _direct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("h2,offset", [(0.5, 0), (0.99, 0), (1.0, 0), (0.5, 20), (0.5, 100),
                                       (0.99, 100)])
def test_guided_search_with_cancelling_sums(c, h2, offset):
    import torch

    from jamma_b200 import engine as eng

    n, m = 600, 500
    rng = np.random.default_rng(100 * c + offset + int(100 * h2))
    z = rng.binomial(2, rng.uniform(0.05, 0.5, 3000), (n, 3000)).astype(np.float64)
    z -= z.mean(0)
    ev, q = np.linalg.eigh(z @ z.T / 3000)
    ev[np.abs(ev) < 1e-10] = 0.0
    assert ev[0] == 0.0 and abs(abs(q[:, 0].sum()) - np.sqrt(n)) < 1e-6 * np.sqrt(n)
    g = rng.binomial(2, rng.uniform(0.01, 0.05, (m, 1)), (m, n)).astype(np.float64)
    u = q @ (rng.standard_normal((n, 2)) * np.sqrt(ev)[:, None])
    y = np.sqrt(h2) * u / u.std(0) + np.sqrt(1 - h2) * rng.standard_normal((n, 2))
    y += g[: m // 2].T @ (0.1 * rng.standard_normal((m // 2, 2)))
    y += offset * y.std(0)
    w = np.column_stack([np.ones(n), rng.standard_normal((n, c - 1)) + offset])
    cohort = eng.DeviceCohort(ev, q, w, y, 4)
    utg = eng.rotate(cohort.U, torch.from_numpy(g).cuda())
    guided = {k: v.cpu().numpy() for k, v in cohort.associate_rotated(utg).items()}
    direct = _direct(cohort, utg)
    for k, p_key in (("lambda_mle", "p_lrt"), ("lambda_remle", "p_wald")):
        a, b = guided[k], direct[k]
        np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
        rel = np.abs(a - b) / b
        # Every decision is the direct search's, but for REML decisions within the rounding of
        # the ones row's sums, which the two forms take from products of different shapes: a
        # few 1e-13 of a log-likelihood against differences of 1e-9 and more.
        assert np.mean(rel <= 1e-13) >= (0.999 if k == "lambda_mle" else 0.99), (k, rel.max())
        # such a decision is one of the last, of brackets of 1e-4
        assert rel.max() <= 1e-4, (k, rel.max())
        # p from the same sums at the same lambda: the same bits but for lambda; at another one,
        # |dlog p| <= (1 + chi2 / 2) |dlog chi2| and |dlog chi2| <= 2 |dlog lambda|
        pa, pb = guided[p_key], direct[p_key]
        dp = np.abs(np.log(pa) - np.log(pb))
        assert np.all(dp <= 1e-9 + 2 * rel * (1 - np.log(pb)) * (rel > 1e-13)), (p_key, dp.max())
    same = np.abs(guided["lambda_remle"] / direct["lambda_remle"] - 1) <= 1e-13
    for k in ("beta", "se"):
        np.testing.assert_allclose(guided[k][same], direct[k][same], rtol=1e-10, atol=0)


@pytest.mark.parametrize("c", [1, 4])
def test_a_pair_does_not_depend_on_the_other_pairs_of_its_chunk(c):
    """Genotypes within rounding of the covariates' span: every grid decision is a matter of
    rounding and left open, by few pairs of a chunk (one CTA each) or by many (one warp each)."""
    import torch

    from jamma_b200 import engine as eng

    n = 800
    rng = np.random.default_rng(c)
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    w = np.column_stack([np.ones(n), rng.standard_normal((n, c - 1))])
    cohort = eng.DeviceCohort(np.sort(rng.gamma(0.7, 0.5, n)), q, w, rng.standard_normal(n), 2)
    utg = torch.from_numpy(rng.uniform(0.3, 1.7, (1500, 1))).cuda() * cohort.UtW[:1]
    utg = utg.contiguous()
    many = {k: v.cpu().numpy()[:, :150] for k, v in cohort.associate_rotated(utg).items()}
    few = {k: v.cpu().numpy() for k, v in cohort.associate_rotated(utg[:150].contiguous()).items()}
    for k in few:
        np.testing.assert_array_equal(many[k], few[k], err_msg=k)


@pytest.mark.parametrize("smallest,guided", [(0.0, True), (-9e-7, True), (-1.1e-6, False),
                                             (-4.9e-6, False)])
def test_no_guided_search_beside_a_pole(smallest, guided):
    """A negative eigenvalue whose weight has its pole just above lambda = 1e5, where the
    expansions over wide brackets lose digits: the search is direct."""
    from jamma_b200 import engine as eng

    n = 500
    rng = np.random.default_rng(0)
    ev = np.sort(rng.gamma(0.7, 0.5, n))
    ev[0] = smallest
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    cohort = eng.DeviceCohort(ev, q, None, rng.standard_normal(n), 4, n_grid=16)
    assert cohort.guided is guided
