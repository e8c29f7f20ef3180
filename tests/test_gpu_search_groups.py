"""The series search at group edges: pair counts around the pairs of a warp (8 for one
covariate column, 4 for more), grid sizes that do not fill the group's lanes, against the
plain FP64 search on the same rotated chunk.  Grids have at least 16 points: their golden
brackets are at most 3.1 wide in log lambda, where the degree-24 bracket expansions truncate
below 1e-15 (Bernstein ellipse parameter above 4)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("m,phi,n_grid", [(1, 1, 50), (7, 1, 50), (9, 1, 18), (5, 3, 17), (33, 2, 51)])
def test_series_search_matches_direct_search_at_group_edges(c, m, phi, n_grid):
    import torch

    from jamma_b200 import engine as eng

    n = 700
    rng = np.random.default_rng(100 * c + m)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    ev = np.sort(rng.gamma(1.0, 1.0, n))
    w = np.column_stack([np.ones(n), rng.standard_normal((n, c - 1))])
    y = q @ (rng.standard_normal((n, phi)) * np.sqrt(ev)[:, None]) + rng.standard_normal((n, phi))
    g = torch.from_numpy(rng.binomial(2, 0.3, (m, n)).astype(np.float64)).cuda()
    outs = []
    for precision in ("fp64", "mixed"):
        cohort = eng.DeviceCohort(ev, q, w, y, 4, n_grid=n_grid, precision=precision)
        outs.append({k: v.cpu().numpy() for k, v in
                     cohort.associate_rotated(eng.rotate(cohort.U, g)).items()})
    plain, series = outs
    # both searches end within the same golden bracket; a step may resolve a near tie apart
    for k in ("lambda_remle", "lambda_mle"):
        np.testing.assert_allclose(series[k], plain[k], rtol=1e-4)
    # at the optimum the likelihood is flat, so the bracket's width does not show in it
    for k in ("logl_h1", "logl_mle"):
        np.testing.assert_allclose(series[k], plain[k], rtol=1e-10)
    for k in ("p_wald", "p_lrt", "p_score"):
        np.testing.assert_allclose(series[k], plain[k], rtol=1e-5)
