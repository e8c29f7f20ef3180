"""The FP64 form's rotation of calls outside the ordinary chunk: no SNPs at all, and a
first rotation that is captured but not replayed."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [1, 2, 3, 4])
def test_no_snps_give_empty_results(mode):
    import torch

    from jamma_b200 import engine as eng

    n = 64
    rng = np.random.default_rng(mode)
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    cohort = eng.DeviceCohort(np.arange(n) / n, q, None, rng.standard_normal((n, 2)), mode)
    codes = torch.empty((0, cohort.code_ld), dtype=torch.int8, device="cuda")
    out = cohort.associate_codes(codes, torch.empty(0, dtype=torch.float64, device="cuda"))
    assert {k: tuple(v.shape) for k, v in out.items()} == {k: (2, 0) for k in eng.MODE_KEYS[mode]}
    assert cohort.rotate_status() == 0


def test_the_first_rotation_may_be_captured():
    """A captured first rotation runs only when it is replayed: an eager one after the capture
    finds the cohort's planes all the same."""
    import torch

    from jamma_b200 import engine as eng

    n, m = 200, 40
    rng = np.random.default_rng(0)
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    cohort = eng.DeviceCohort(np.arange(n) / n, q, None, rng.standard_normal(n), 1)
    g = rng.integers(0, 3, (m, n))
    codes = torch.zeros((m, cohort.code_ld), dtype=torch.int8, device="cuda")
    codes[:, :n] = torch.from_numpy(g).cuda()
    mu = torch.ones(m, dtype=torch.float64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        cohort.rotate_codes_f64(codes, mu, True)
    got = cohort.rotate_codes_f64(codes, mu, True).cpu().numpy()
    np.testing.assert_allclose(got, g @ q, rtol=0, atol=1e-12)
