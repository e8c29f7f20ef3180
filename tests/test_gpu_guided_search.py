"""The FP64 form's guided search against the search of direct evaluations (precision 0) on the
same cohort and rotated chunk: sample counts around the guided form's lower limit and its
staging tile (512 samples), every covariate count, spectra and phenotypes with flat
likelihoods (open decisions, few and many) and an all-zero genotype."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _direct(cohort, utg):
    from jamma_b200 import _native
    from jamma_b200.device import ptr, stream_handle

    c = cohort
    assert c.guided and c._form == 3
    c._form = 0
    _native.call("jb_lmm_prepare", c.mode, 0, c.n, c.c, c.phi, ptr(c.evals), ptr(c.UtW), c.n,
                 ptr(c.Uty), c.n, ptr(c.lam0), c.l_min, c.l_max, c.n_grid, ptr(c.ws), c.ws.numel(),
                 stream_handle())
    return {k: v.cpu().numpy() for k, v in c.associate_rotated(utg).items()}


@pytest.mark.parametrize("n,c,mode", [(400, 1, 4), (511, 2, 4), (513, 3, 1), (1025, 4, 4),
                                      (1030, 1, 2), (700, 2, 3), (2049, 1, 4)])
@pytest.mark.parametrize("scale", [0.0, 1.0, 1000.0])  # polygenic part: none, as the noise, all
def test_guided_search_takes_the_decisions_of_direct_evaluations(n, c, mode, scale):
    import torch

    from jamma_b200 import engine as eng

    rng = np.random.default_rng(n + c)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    ev = np.sort(rng.gamma(0.7, 0.5, n))
    ev[0] = 0.0
    w = np.column_stack([np.ones(n), rng.standard_normal((n, c - 1))])
    y = q @ (rng.standard_normal((n, 2)) * np.sqrt(scale * ev)[:, None]) + rng.standard_normal((n, 2))
    m = 1203 if scale == 1.0 else 300
    g = rng.binomial(2, rng.uniform(0.05, 0.95, (m, 1)), (m, n)).astype(np.float64)
    g[3] = 0.0
    g[4] = 0.05 * g[4] + y[:, 0]  # an SNP that explains almost everything
    cohort = eng.DeviceCohort(ev, q, w, y, mode)
    utg = eng.rotate(cohort.U, torch.from_numpy(g).cuda())
    guided = {k: v.cpu().numpy() for k, v in cohort.associate_rotated(utg).items()}
    direct = _direct(cohort, utg)
    for k in direct:
        np.testing.assert_array_equal(np.isnan(guided[k]), np.isnan(direct[k]), err_msg=k)
    ok = np.ones(m, bool)
    ok[4] = False  # its likelihood is dominated by the rounding of P_yy: compared above only
    for k in direct:
        a, b = guided[k][:, ok], direct[k][:, ok]
        fin = np.isfinite(b)
        rel = np.abs(a - b)[fin] / np.maximum(np.abs(b[fin]), 1e-300)
        if k.startswith("lambda"):
            # the same bits, but for decisions within the rounding of the ones row's sums
            # (REML), which the two forms take from products of different shapes
            assert np.mean(rel <= 1e-13) >= (0.999 if k == "lambda_mle" else 0.95), (k, rel.max())
            assert rel.max() <= 1e-4, k
        elif k.startswith("logl"):
            assert rel.max() <= 1e-12, (k, rel.max())
        elif k == "p_score":
            assert rel.max() <= 1e-8, (k, rel.max())
